"""Scratch of the adjoint of the mixed term (GPU): bounded by bytes, whatever the image size and field count, and by
what the device has left."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,K,most", [(2048, 20, 512 << 20), (4300, 5, 512 << 20), (256, 40, 512 << 20)])
def test_mixed_transpose_scratch(cuda, side, K, most):
    """2048: 35 MB a field, 15 per launch; 4300: 150 MB a field, 3 per launch; 256: 32 fields per launch."""
    from test_gpu_pcg_sizes import _adjoint
    adj = _adjoint(cuda, side, 64)
    g = torch.Generator(device=cuda).manual_seed(side)
    lam = torch.randn((adj.L.n_nodes, 2, K), generator=g, device=cuda)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated(cuda)
    torch.cuda.reset_peak_memory_stats(cuda)
    out = adj.mixed_T(lam)
    torch.cuda.synchronize()
    scratch = torch.cuda.max_memory_allocated(cuda) - before - out.numel() * 4
    assert scratch <= most + (4 << 20)                   # and the fields themselves
    # each field as by itself, to the order of the atomic additions (FP32, at most 64 terms per coefficient)
    for k in (0, K - 1):
        one = adj.mixed_T(lam[:, :, k:k + 1])[0]
        assert float((out[k] - one).abs().max()) <= 1e-5 * float(one.abs().max())


def test_fewer_fields_where_the_device_has_no_room(cuda):
    """A limit that leaves room for the result and two fields: the call that fits one at a time still runs."""
    from test_gpu_pcg_sizes import _adjoint
    side, K = 1500, 16
    adj = _adjoint(cuda, side, 64)
    g = torch.Generator(device=cuda).manual_seed(1)
    lam = torch.randn((adj.L.n_nodes, 2, K), generator=g, device=cuda)
    want = adj.mixed_T(lam)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    field = 4 * adj.L.cpitch * (2 * side + 64)
    room = torch.cuda.memory_reserved(cuda) + want.numel() * 4 + 2 * field + (44 << 20)
    total = torch.cuda.get_device_properties(cuda).total_memory
    torch.cuda.set_per_process_memory_fraction(room / total, cuda)
    try:
        got = adj.mixed_T(lam)
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, cuda)
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())

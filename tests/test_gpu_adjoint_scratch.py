"""Scratch of the adjoint of the mixed term (GPU): bounded by bytes, whatever the image size and field count."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,K,most", [(2048, 9, 128 << 20), (4300, 2, 152 << 20), (256, 40, 128 << 20)])
def test_mixed_transpose_scratch(cuda, side, K, most):
    """2048: 35 MB a field, 3 per launch; 4300: 151 MB a field, one per launch; 256: 32 fields per launch."""
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

"""The adjoint's PCG on a large mesh on both sides of the line between vectors on the chip and in memory (GPU).

The residual B - H X in FP64 with the operator's FP32 entries: the stop rule leaves 1e-7 of ||B||, the FP32
product rounds to a few 6e-8 of the row's terms, which cancel at most about 30-fold here: 1e-5.
"""
from __future__ import annotations

import pytest
import torch

from test_gpu_pcg_sizes import _adjoint, _residual

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [32, 33])
def test_columns_on_a_large_mesh(cuda, K):
    from d2ic_gb300 import _lib
    adj = _adjoint(cuda, 1112, 2, roi=1098)
    n = adj.L.n_nodes
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    per_sm = -(-n // sms)
    assert 3875 // 2 < per_sm <= 3875                  # one column per launch fits
    assert (_lib.load().d2ic_pcg_plan(n, K, sms, None) == 0) == (K > 32)
    g = torch.Generator(device=cuda).manual_seed(K)
    B = torch.randn((n, 2, K), generator=g, device=cuda, dtype=torch.float64) * adj.active[:, None, None]
    B[:, :, 3] = 0.0
    X = adj.solve(B)
    assert float(_residual(adj, X, B).max()) <= 1e-5
    assert not X[:, :, 3].any() and 0 < adj.last_iters < 2000

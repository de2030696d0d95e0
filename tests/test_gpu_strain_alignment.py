"""Linearised strain of directions that start between 16-byte boundaries (GPU): a slice of a packed FP64 vector
is contiguous, passes through unchanged, and gives the bits of an aligned copy."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,offset", [(1, 1, 1), (33, 4, 1), (129, 5, 3), (40, 9, 2)])
def test_directions_at_an_odd_offset(cuda, n, K, offset):
    from d2ic_gb300.adjoint import strain_jvp
    rng = np.random.default_rng(n)
    X, u = rng.uniform(0, 40, (n, 2)), rng.normal(0, 0.05, (n, 2))
    idx = rng.integers(0, n, (n, 6)).astype(np.int32)
    deg = rng.integers(1, 7, n).astype(np.int32)
    packed = torch.as_tensor(rng.normal(0, 1, offset + K * n * 2), device=cuda)
    du = packed[offset:].view(K, n, 2)
    assert du.is_contiguous() and du.data_ptr() % 16 == 8 * (offset % 2)
    u = torch.as_tensor(u, device=cuda)
    got = strain_jvp(u, du, X, idx, deg, 15.0)
    assert torch.equal(got, strain_jvp(u, du.clone(), X, idx, deg, 15.0))
    assert torch.isfinite(got).all()

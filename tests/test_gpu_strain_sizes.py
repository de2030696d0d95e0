"""Strain kernels at the edges of their blocks (GPU): node counts around a warp, degrees around the neighbours in
flight, malformed and missing neighbours, direction counts around those of one thread; against the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _graph(n, md, seed):
    rng = np.random.default_rng(seed)
    X = rng.uniform(0, 40, (n, 2)).astype(np.float32)
    deg = rng.integers(min(2, md), md + 1, n).astype(np.int32)
    idx = np.stack([rng.permutation(n)[:md] if n >= md else rng.integers(0, n, md) for _ in range(n)]).astype(np.int32)
    u = (0.01 * X + rng.normal(0, 0.05, (n, 2))).astype(np.float32)
    return X, idx, deg, u


@pytest.mark.parametrize("n,md,gauge", [(1, 1, 0.0), (31, 3, 8.0), (33, 4, 0.0), (64, 5, 20.0), (129, 9, 8.0)])
def test_strain_against_oracle(cuda, n, md, gauge):
    from d2ic_gb300 import _lib
    from d2ic_gb300._lib import ptr
    from oracle.strain import green_lagrange_nodes_lsq
    X, idx, deg, u = _graph(n, md, n)
    T = lambda a: torch.as_tensor(a, device=cuda)
    out = torch.empty((n, 3), dtype=torch.float32, device=cuda)
    args = [T(u), T(X), T(idx), T(deg)]
    _lib.call("d2ic_strain_gl", *[ptr(a) for a in args], n, md, gauge, 1e-8, ptr(out), 0, _lib.stream_handle())
    _, E = green_lagrange_nodes_lsq(u.astype(np.float64), X.astype(np.float64), idx, deg, gauge, float(np.float32(1e-8)))
    want = np.stack([E[:, 0, 0], E[:, 1, 1], E[:, 0, 1]], axis=1)
    # one FP32 rounding of the result; the sums are FP64, their condition is at most 1e6 here
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-7 * max(np.abs(want).max(), 1.0) + 1e-9


@pytest.mark.parametrize("n,md,K", [(31, 4, 1), (33, 3, 3), (127, 8, 4), (129, 9, 5), (40, 6, 9)])
def test_strain_jvp_of_several_directions(cuda, n, md, K):
    from d2ic_gb300.adjoint import strain_jvp
    X, idx, deg, u = _graph(n, md, 100 + n)
    X, u = X.astype(np.float64), u.astype(np.float64)
    du = np.random.default_rng(K).normal(0, 1, (K, n, 2))
    got = strain_jvp(torch.as_tensor(u, device=cuda), torch.as_tensor(du, device=cuda), X, idx, deg, 15.0).cpu().numpy()
    want = np.zeros((K, n, 3))
    for i in range(n):
        j = idx[i, :deg[i]]
        dX = X[j] - X[i]
        w = np.exp(-(dX ** 2).sum(axis=1) / (15.0 + 1e-12) ** 2)
        Ainv = np.linalg.inv(np.einsum("k,ka,kb->ab", w, dX, dX) + 1e-8 * np.eye(2))
        grad = lambda v: np.einsum("ab,k,kb,kc->ca", Ainv, w, dX, v[j] - v[i])
        F = np.eye(2) + grad(u)
        for k in range(K):
            S = grad(du[k]).T @ F
            want[k, i] = S[0, 0], S[1, 1], 0.5 * (S[0, 1] + S[1, 0])
    assert np.abs(got - want).max() <= 1e-7 * max(np.abs(want).max(), 1.0)

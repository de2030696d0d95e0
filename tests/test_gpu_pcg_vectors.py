"""The vectors and sums of the adjoint's PCG on the chip (GPU) against CG with FP64 vectors and the same products.

The FP32 product of d2ic_hessian_apply has the bits of the solver's, so what is compared is the precision of
everything else.  With vectors of 48 bits in place of FP64 a CPU model (block-Jacobi CG, FP32 products, 144 to
3,600 nodes, 1 to 6 columns) ends 8e-12 to 1.4e-10 of the solution's norm away -- an entry of P on the edge of an FP32
rounding -- and with FP32 vectors, 1.6e-7.  A dropped low word of one sum or product lies between.  The bound
is 3e-9; the iteration counts are equal.

Beyond that size CG amplifies the order of the sums alone: FP64 vectors whose sums run in another order end
5e-9 away after 103 iterations on 22,801 nodes.  There the two are compared by their distances from CG
with FP64 products, 1e-7 with FP64 vectors and twice that with FP32 ones, with the same bound.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_pcg_sizes import _adjoint, _residual

pytestmark = pytest.mark.gpu


def _sparse(adj):
    """The operator's FP32 entries as an FP64 matrix over the active nodes' components."""
    n = adj.L.n_nodes
    op = adj.operator()
    blk = op[: n * 256].view(torch.float32).reshape(n, 16, 4).to(torch.float64)
    at = (n * 256 + 255) // 256 * 256
    idx = op[at: at + n * 64].view(torch.int32).reshape(n, 16).long()
    on = (idx >= 0) & adj.active[:, None]
    r = torch.arange(n, device=idx.device)[:, None].expand(n, 16)[on]
    c, b = idx[on], blk[on]
    rows, cols = torch.cat([2 * r, 2 * r, 2 * r + 1, 2 * r + 1]), torch.cat([2 * c, 2 * c + 1, 2 * c, 2 * c + 1])
    vals = torch.cat([b[:, 0], b[:, 1], b[:, 1], b[:, 2]])
    return torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (2 * n, 2 * n)).coalesce().to_sparse_csr()


def _cg64(adj, B, rtol, iters=400, matrix=None):
    """CG with FP64 vectors and the FP32 products of d2ic_hessian_apply, or the FP64 products of a matrix.  P is
    scaled by a power of two (exact) for the FP32 product, so that it stays in FP32's range."""
    M = adj.Minv
    on = adj.active[:, None, None]
    s = 2.0 ** -round(float(torch.log2(M.abs().max())) / 2)
    pre = lambda v: torch.einsum("nij,njk->nik", M, v)
    dot = lambda a, b: (a * b).sum(dim=(0, 1))
    X = torch.zeros_like(B)
    R = B * on
    Z = pre(R)
    P = Z.clone()
    rz, bb = dot(R, Z), dot(R, R)
    Y = torch.empty(B.shape, dtype=torch.float32, device=B.device)
    for it in range(1, iters + 1):
        if matrix is None:
            adj.apply((P * s).to(torch.float32), Y)
            AP = Y.to(torch.float64) / s * on
        else:
            AP = (matrix @ P.reshape(-1, P.shape[2])).reshape(P.shape) * on
        pap = dot(P, AP)
        a = torch.where(pap > 0, rz / pap, 0.0)
        X += a * P
        R -= a * AP
        if bool((dot(R, R).sqrt() <= rtol * bb.sqrt().clamp(min=1e-300)).all()):
            return X, it
        Z = pre(R)
        now = dot(R, Z)
        P = Z + torch.where(rz > 0, now / rz, 0.0) * P
        rz = now
    raise AssertionError("no convergence")


def _rhs(adj, K, device):
    g = torch.Generator(device=device).manual_seed(K)
    return torch.randn((adj.L.n_nodes, 2, K), generator=g, device=device, dtype=torch.float64) * adj.active[:, None, None]


@pytest.mark.parametrize("side,element,K", [
    (60, 16, 1),          # one block
    (300, 16, 3),         # 361 nodes, several blocks of few nodes
    (400, 10, 1),
    (400, 10, 6),         # columns that do not divide a warp
    (530, 10, 64),        # one full launch of columns
    (530, 10, 67),        # two launches, the second of three columns
    (900, 6, 130),        # operator and preconditioner read from memory
])
def test_solution_of_fp64_vectors(cuda, side, element, K):
    adj = _adjoint(cuda, side, element)
    B = _rhs(adj, K, cuda)
    want, its = _cg64(adj, B, 1e-11)
    X = adj.solve(B, rtol=1e-11)
    norm = lambda v: v.flatten(0, 1).norm(dim=0)
    if adj.L.n_nodes <= 3600:
        excess = norm(X - want) / norm(want)
    else:
        exact, _ = _cg64(adj, B, 1e-13, matrix=_sparse(adj))
        excess = (norm(X - exact) - norm(want - exact)) / norm(exact)
    assert float(excess.max()) <= 3e-9, float(excess.max())
    assert adj.last_iters == its


def _scaled(device, side, element, scale, K):
    """The linearisation of a frame whose grey levels are multiplied by a power of two, without springs."""
    import d2ic_gb300 as d2
    from d2ic_gb300.adjoint import ImplicitAdjoint
    from d2ic_gb300.engine import FrameLayout, FrameSlot
    from d2ic_gb300.synthetic import rect_mask
    rng = np.random.default_rng(side)
    image = torch.as_tensor(128 + 40 * rng.standard_normal((side, side)), dtype=torch.float32) * scale
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 12, side - 12), element)
    pix = d2.build_pixel_assets(mesh, image.numpy(), 1.0, assets.roi_mask)
    layout = FrameLayout(pix, mesh.nodes_xy.shape[0], image.numpy(), "cubic", device)
    slot = FrameSlot(layout, 1)
    slot.load_image(image.numpy())
    adj = ImplicitAdjoint(slot, torch.zeros((layout.n_nodes, 2), device=device), 0.0, exact=False)
    return adj, _rhs(adj, K, device)


@pytest.mark.parametrize("exponent", [-62, -40, 0, 49])
@pytest.mark.parametrize("side,K", [(150, 2), (400, 5)])
def test_grey_levels_of_any_size(cuda, side, K, exponent):
    """Operator entries from 1e-37 to 1e31: FP64 vectors hold the inverse blocks, and so do these."""
    adj, B = _scaled(cuda, side, 12, 2.0 ** exponent, K)
    X = adj.solve(B, rtol=1e-9)
    assert torch.isfinite(X).all() and 0 < adj.last_iters < 400
    assert float(_residual(adj, X, B).max()) <= 1e-5
    want, its = _cg64(adj, B, 1e-9)
    err = (X - want).flatten(0, 1).norm(dim=0) / want.flatten(0, 1).norm(dim=0)
    assert float(err.max()) <= 3e-9, float(err.max())
    assert adj.last_iters == its

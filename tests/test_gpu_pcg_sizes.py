"""The adjoint's PCG over its plans (GPU): one block, blocks with grid sums, several launches of columns,
and the form with its vectors in memory for meshes beyond the chip.

The solution is judged by its residual B - H X in FP64 with the operator's own FP32 entries: the stop
rule leaves 1e-7, the FP32 product of a row of at most 16 blocks rounds to 32 * 6e-8 of the row's terms;
1e-5 covers both with the rows' cancellation.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _adjoint(device, side, element, roi=None):
    import d2ic_gb300 as d2
    from d2ic_gb300.adjoint import ImplicitAdjoint
    from d2ic_gb300.engine import FrameLayout, FrameSlot
    from d2ic_gb300.pixel_assets import build_pixel_assets_device
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence_device
    ref, frames = speckle_sequence_device(side, side, [Translation(0.2, -0.1)], seed=7, noise_seeds=[1, 2], device=device,
                                          u8=False)
    inner = side - 12 if roi is None else roi
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, inner, inner), element)
    pix = build_pixel_assets_device(mesh, np.empty((side, side), np.uint8), 1.0, assets.roi_mask)
    layout = FrameLayout(pix, mesh.nodes_xy.shape[0], ref, "cubic", device)
    slot = FrameSlot(layout, 1)
    slot.load_image(frames[0])
    u = torch.zeros((layout.n_nodes, 2), device=device) + torch.tensor([0.2, -0.1], device=device)
    return ImplicitAdjoint(slot, u, 0.1)


def _residual(adj, X, B):
    # the operator's entries: (column node, block) of each node, packed
    n = adj.L.n_nodes
    op = adj.operator()
    blk = op[: n * 256].view(torch.float32).reshape(n, 16, 4).to(torch.float64)
    at = (n * 256 + 255) // 256 * 256
    idx = op[at: at + n * 64].view(torch.int32).reshape(n, 16).long()
    on = (idx >= 0)[:, :, None].to(torch.float64)
    R = B.clone()
    for q in range(16):
        v = X[idx[:, q].clamp(min=0)] * on[:, q, :, None]
        b = blk[:, q]
        R[:, 0] -= b[:, 0:1] * v[:, 0] + b[:, 1:2] * v[:, 1]
        R[:, 1] -= b[:, 1:2] * v[:, 0] + b[:, 2:3] * v[:, 1]
    R *= adj.active[:, None, None]
    return R.flatten(0, 1).norm(dim=0) / B.flatten(0, 1).norm(dim=0).clamp(min=1e-300)


@pytest.mark.parametrize("side,element,K", [
    (60, 16, 1),          # 16 nodes: one block
    (400, 10, 1),         # 41 x 41 nodes: one block, several nodes per thread
    (400, 10, 6),         # several blocks, columns that do not divide a warp
    (530, 10, 64),        # one full launch of columns
    (530, 10, 67),        # two launches, the second of three columns
    (900, 6, 130),        # 22,801 nodes: fewer columns per launch
])
def test_columns_converge_in_every_plan(cuda, side, element, K):
    adj = _adjoint(cuda, side, element)
    g = torch.Generator(device=cuda).manual_seed(K)
    B = torch.randn((adj.L.n_nodes, 2, K), generator=g, device=cuda, dtype=torch.float64) * adj.active[:, None, None]
    B *= torch.logspace(-30, 20, K, dtype=torch.float64, device=cuda)     # columns of very different size
    if K > 2:
        B[:, :, 1] = 0.0
    X = adj.solve(B)
    r = _residual(adj, X, B)
    assert float(r.max()) <= 1e-5, float(r.max())
    assert 0 < adj.last_iters < 2000
    if K > 2:
        assert not X[:, :, 1].any()
    assert not X[~adj.active].any()


def test_mesh_beyond_the_chip(cuda):
    """More than 547,000 nodes: the vectors stay in memory."""
    adj = _adjoint(cuda, 1604, 2, roi=1590)
    assert adj.L.n_nodes > 560_000
    g = torch.Generator(device=cuda).manual_seed(3)
    B = torch.randn((adj.L.n_nodes, 2, 1), generator=g, device=cuda, dtype=torch.float64) * adj.active[:, None, None]
    X = adj.solve(B)
    assert float(_residual(adj, X, B).max()) <= 1e-5


def test_iteration_limit(cuda):
    adj = _adjoint(cuda, 400, 10)
    B = torch.ones((adj.L.n_nodes, 2, 3), device=cuda, dtype=torch.float64) * adj.active[:, None, None]
    assert not adj.solve(B, max_iter=0).any() and adj.last_iters == 0
    adj.solve(B, rtol=0.0, max_iter=5)
    assert adj.last_iters == 5


@pytest.mark.parametrize("side,element", [(60, 16), (205, 13), (260, 32)])
def test_preconditioner_inverts_the_diagonal_blocks(cuda, side, element):
    """Minv of every node is the inverse of the 2x2 diagonal block of H (chunk blocks plus springs, summed in
    FP64 here); nodes of no element are inactive.  The blocks are FP32 sums of at most 16 chunks and 8
    springs: 24 * 6e-8, times the blocks' condition."""
    adj = _adjoint(cuda, side, element)
    L = adj.L
    h = adj.hess.cpu().numpy().reshape(-1, 32)[: L.n_chunks].astype(np.float64)
    cn = L.chunk_nodes.cpu().numpy()
    D = np.zeros((L.n_nodes, 2, 2))
    for a in range(4):
        p = 3 * (a * 4 - (a * (a - 1)) // 2)
        for (i, j), q in (((0, 0), 0), ((0, 1), 1), ((1, 0), 1), ((1, 1), 2)):
            np.add.at(D[:, i, j], cn[:, a], h[:, p + q] * adj.inv_np)
    w = np.where(L.nbr_index.cpu().numpy() >= 0, L.nbr_weight.cpu().numpy(), 0.0).astype(np.float64).sum(axis=0)
    D[:, 0, 0] += adj.alpha * w
    D[:, 1, 1] += adj.alpha * w
    active = adj.active.cpu().numpy()
    used = np.zeros(L.n_nodes, bool)
    used[cn.ravel()] = True
    assert np.array_equal(active, used | (w > 0))
    M = adj.Minv.cpu().numpy()
    assert not M[~active].any()
    cond = np.linalg.cond(D[active]).max()
    assert np.abs(M[active] @ D[active] - np.eye(2)).max() <= 24 * 6e-8 * cond * 4

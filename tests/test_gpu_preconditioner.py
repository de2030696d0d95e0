"""The adjoint's block-Jacobi preconditioner against FP64 sums of the chunks' FP32 blocks (GPU)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(device, side, element, image, alpha):
    import d2ic_gb300 as d2
    from d2ic_gb300.adjoint import ImplicitAdjoint
    from d2ic_gb300.engine import FrameLayout, FrameSlot
    from d2ic_gb300.synthetic import rect_mask
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 8, side - 8), element)
    pix = d2.build_pixel_assets(mesh, image, 1.0, assets.roi_mask)
    layout = FrameLayout(pix, mesh.nodes_xy.shape[0], image, "cubic", device)
    slot = FrameSlot(layout, 1)
    slot.load_image(image)
    u = torch.full((layout.n_nodes, 2), 0.3, device=device)
    return ImplicitAdjoint(slot, u, alpha, exact=False)


def _blocks(adj):
    L = adj.L
    h = adj.hess.cpu().numpy().reshape(-1, 32)[: L.n_chunks]
    cn = L.chunk_nodes.cpu().numpy()
    D = np.zeros((L.n_nodes, 3))
    for a in range(4):
        p = 3 * (a * 4 - (a * (a - 1)) // 2)
        np.add.at(D, cn[:, a], (h[:, p:p + 3] * np.float32(adj.inv_np)).astype(np.float64))
    w = np.where(L.nbr_index.cpu().numpy() >= 0, L.nbr_weight.cpu().numpy(), 0.0).astype(np.float64).sum(axis=0)
    D[:, 0] += float(np.float32(adj.alpha)) * w
    D[:, 2] += float(np.float32(adj.alpha)) * w
    return D, D[:, 0] * D[:, 2] - D[:, 1] ** 2


@pytest.mark.parametrize("side,element,alpha", [(60, 16, 0.1), (205, 13, 0.1), (260, 40, 0.5), (131, 9, 0.0)])
def test_blocks_are_fp64_sums(cuda, side, element, alpha):
    """At most 4 x 16 chunk blocks and 8 springs, each addition rounded to 1.1e-16, times the condition."""
    rng = np.random.default_rng(side)
    adj = _case(cuda, side, element, (128 + 40 * rng.standard_normal((side, side))).astype(np.float32), alpha)
    D, det = _blocks(adj)
    on = (np.abs(D).sum(axis=1) > 0) & (det > 0)
    assert np.array_equal(adj.active.cpu().numpy(), on) and on.any()
    M = adj.Minv.cpu().numpy()
    assert not M[~on].any()
    want = np.stack([D[:, 2], -D[:, 1], -D[:, 1], D[:, 0]], axis=1)[on].reshape(-1, 2, 2) / det[on][:, None, None]
    cond = (np.abs(D[on]).max(axis=1) ** 2 / det[on]).max()
    assert np.abs(M[on] - want).max() <= 72 * 1.2e-16 * 8 * cond * np.abs(want).max()


@pytest.mark.parametrize("side,element", [(96, 12), (150, 16)])
def test_nodes_of_stripes_along_the_diagonal(cuda, side, element):
    """Without springs and with grey levels of x + y only, the blocks are singular but for the rounding of the
    chunks' sums: which nodes are active is decided by the FP64 determinant of the FP32 chunk blocks."""
    y, x = np.mgrid[:side, :side]
    image = (128 + 100 * np.sin(0.35 * (x + y))).astype(np.float32)
    adj = _case(cuda, side, element, image, 0.0)
    D, det = _blocks(adj)
    clear = np.abs(det) > 1e-13 * D[:, 0] * D[:, 2]        # beyond the order of the additions
    on = (np.abs(D).sum(axis=1) > 0) & (det > 0)
    got = adj.active.cpu().numpy()
    assert clear.sum() > got.size // 2 and (det[clear] < 1e-4 * (D[:, 0] * D[:, 2])[clear]).any()
    assert np.array_equal(got[clear], on[clear])

"""Pixels whose local coordinates lie outside their element (GPU), as a caller's own shape functions may put them:
their displacement is no mean of the nodes', so their stencils may leave the window that a chunk's nodes span."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(side, element, stretch):
    import d2ic_gb300 as d2
    from d2ic_gb300.pixel_assets import shape_functions
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    from oracle import objective, pixels
    ref, frames = speckle_sequence(side, side, [Translation(0.35, -0.25)], seed=side, noise_seeds=[1, 2])
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 30, side - 30), element)
    pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
    xe = stretch * np.asarray(pix.xi_eta)
    N = shape_functions(xe[:, 0], xe[:, 1])
    pix.xi_eta, pix.pixel_shapeN = xe, N
    assets = replace(assets, pixel_data=pix)
    oa = pixels.build_pixel_assets(np.asarray(mesh.nodes_xy), np.asarray(mesh.elements), side, side, assets.roi_mask)
    pb = objective.Problem.build(ref, frames[0], oa, "cubic")
    assert pb.pixel_shapeN.shape == N.shape
    pb.pixel_shapeN = N
    u = np.random.default_rng(7).normal(0.0, 1.5, (mesh.nodes_xy.shape[0], 2)).astype(np.float32)
    return ref, frames[0], mesh, assets, pb, u


@pytest.mark.parametrize("side,element,stretch", [(120, 8, 1.0), (120, 8, 2.5), (110, 14, 3.0)])
def test_local_refinement(cuda, side, element, stretch):
    import d2ic_gb300 as d2
    from oracle import local_gn
    ref, image, mesh, assets, pb, u0 = _case(side, element, stretch)
    cfg = d2.MeshDICConfig(max_iters=2, tol=1e-3, reg_strength=0.1, save_history=True)
    dic = d2.DICMeshBased(mesh, d2.LocalGaussNewtonSolver(device=cuda), cfg)
    dic.prepare(ref, assets)
    dic.set_initial_guess(u0)
    res = dic.run(image)
    want, hist = local_gn.local_sweeps(u0, pb, 1e-3, 0.2, 0.1, 0.5, 2)
    assert np.abs(np.asarray(res.u_nodal, np.float64) - want).max() <= 1e-3
    assert np.allclose(np.asarray(res.history), hist, rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("side,element,stretch", [(120, 8, 1.0), (120, 8, 2.5), (110, 14, 3.0)])
def test_mixed_term(cuda, side, element, stretch):
    """Windows (20 images at a time) and global memory (one image): the same bits, and the FP64 oracle's."""
    from d2ic_gb300.adjoint import ImplicitAdjoint
    from d2ic_gb300.engine import FrameLayout, FrameSlot
    from oracle import adjoint as oadj
    ref, image, mesh, assets, pb, u = _case(side, element, stretch)
    layout = FrameLayout(assets.pixel_data, mesh.nodes_xy.shape[0], ref, "cubic", cuda)
    slot = FrameSlot(layout, 1)
    slot.load_image(image)
    adj = ImplicitAdjoint(slot, u, 0.1)
    dI = np.random.default_rng(3).normal(0, 1, (20, side, side)).astype(np.float32)
    many = adj.mixed(torch.as_tensor(dI, device=cuda))
    one = adj.mixed(torch.as_tensor(dI[:1], device=cuda))
    assert torch.equal(many[:, :, 0], one[:, :, 0])
    want = np.asarray(oadj.mixed_term(u.astype(np.float64), pb, dI[0].astype(np.float64))).reshape(-1, 2)
    got = one[:, :, 0].cpu().numpy()
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()

"""Local Gauss-Newton sweeps where chunks' windows fit shared memory, do not fit or leave the image (GPU), and
more sweeps than one history launch takes, against the FP64 oracle sweeps."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,element,spread,sweeps", [
    (97, 8, 0.2, 3),          # 64-pixel chunks
    (131, 41, 0.2, 2),        # several chunks per element, wide windows
    (96, 16, 6.0, 2),         # nodes of an element far apart: windows too large, partly outside the image
    (80, 13, 0.1, 35),        # three history launches
])
def test_sweeps_match_oracle(cuda, side, element, spread, sweeps):
    import d2ic_gb300 as d2
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    from oracle import local_gn, objective, pixels
    ref, frames = speckle_sequence(side, side, [Translation(0.35, -0.25)], seed=side, noise_seeds=[side, side + 1])
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 6, side - 6), element)
    assets = replace(assets, pixel_data=d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask))
    cfg = d2.MeshDICConfig(max_iters=sweeps, tol=1e-3, reg_strength=0.1, save_history=True)
    dic = d2.DICMeshBased(mesh, d2.LocalGaussNewtonSolver(device=cuda), cfg)
    dic.prepare(ref, assets)
    u0 = np.random.default_rng(7).normal(0.0, spread, (mesh.nodes_xy.shape[0], 2)).astype(np.float32)
    dic.set_initial_guess(u0)
    res = dic.run(frames[0])
    oa = pixels.build_pixel_assets(np.asarray(mesh.nodes_xy), np.asarray(mesh.elements), side, side, assets.roi_mask)
    pb = objective.Problem.build(ref, frames[0], oa, interpolation="cubic")
    u_ref, h_ref = local_gn.local_sweeps(u0, pb, 1e-3, 0.2, 0.1, 0.5, sweeps)
    assert np.abs(np.asarray(res.u_nodal, np.float64) - u_ref).max() <= 1e-3         # nodal tolerance, px
    assert np.allclose(np.asarray(res.history), h_ref, rtol=1e-3, atol=1e-6)


@pytest.mark.parametrize("H,W", [(1, 1), (2, 130), (133, 3), (260, 197)])
def test_gradient_coefficients_are_those_of_the_gradient_images(cuda, H, W):
    from d2ic_gb300 import _lib
    from d2ic_gb300._lib import ptr
    from d2ic_gb300.engine import PAD, prepare_coefficients
    img = torch.rand((H, W), device=cuda) * 255
    gx, gy = torch.empty_like(img), torch.empty_like(img)
    _lib.call("d2ic_central_gradient", ptr(img), H, W, ptr(gx), ptr(gy), _lib.stream_handle())
    want = [prepare_coefficients(x, _lib.INTERP_CUBIC) for x in (img, gx, gy)]
    got = [torch.zeros_like(w) for w in want]
    _lib.call("d2ic_bspline_prefilter_gradients", ptr(img), H, W, PAD, want[0].shape[1], *[ptr(g) for g in got],
              _lib.stream_handle())
    for g, w in zip(got, want):
        assert torch.equal(g[:, :W + 2 * PAD], w[:, :W + 2 * PAD])

"""Local refinement without sweeps (GPU): the start is the result, whatever the count below one."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweeps", [0, -1, -2])
@pytest.mark.parametrize("interp", ["cubic", "linear"])
def test_no_sweeps_return_the_start(cuda, sweeps, interp):
    import d2ic_gb300 as d2
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    ref, frames = speckle_sequence(64, 64, [Translation(0.3, -0.2)], seed=1, noise_seeds=[1, 2])
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(64, 64, 48, 48), 16)
    assets = replace(assets, pixel_data=d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask))
    cfg = d2.MeshDICConfig(max_iters=sweeps, tol=1e-3, reg_strength=0.1, save_history=True)
    dic = d2.DICMeshBased(mesh, d2.LocalGaussNewtonSolver(interpolation=interp, device=cuda), cfg)
    dic.prepare(ref, assets)
    u0 = np.random.default_rng(2).normal(0.0, 0.3, (mesh.nodes_xy.shape[0], 2)).astype(np.float32)
    dic.set_initial_guess(u0)
    res = dic.run(frames[0])
    assert np.array_equal(np.asarray(res.u_nodal), u0)
    assert len(res.history) == 0

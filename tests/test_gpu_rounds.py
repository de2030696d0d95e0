"""Rounds of the CG engine at the edges of its work split (GPU).

The split of a round over the grid -- a supergroup reduced in one block or through global partials,
blocks with and without a lighter share of the chunks, a control step on a warp of its own or on the
one that completes the frame -- depends on the number of node groups and chunks against the warps of
the grid.  Every partial has its own slot and every sum a fixed order, so a solve gives the same bits
on every grid; one evaluation is compared with the FP64 oracle.
"""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,element,interp", [
    (40, 16, "cubic"),        # 9 nodes: one group
    (354, 16, "cubic"),       # 23 x 23 nodes: 17 groups, the second supergroup has one
    (250, 8, "cubic"),        # 32 x 32 nodes: 32 groups, two full supergroups; 64-pixel chunks
    (257, 11, "linear"),      # odd image and element sizes
    (300, 32, "cubic"),       # several chunks per element: 16 slots per node
])
def test_grids_give_the_same_bits(cuda, side, element, interp):
    import d2ic_gb300 as d2
    from d2ic_gb300.engine import Engine, FrameLayout, FrameSlot, descriptors_to_device
    from d2ic_gb300.synthetic import Affine, rect_mask, speckle_sequence
    from oracle import objective, pixels
    ref, frames = speckle_sequence(side, side, [Affine([[0.004, 0.001], [0, -0.003]], [0.4, -0.3], [side / 2] * 2)],
                                   seed=81, noise_seeds=[81, 82])
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 12, side - 12), element)
    pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
    n_nodes = mesh.nodes_xy.shape[0]
    layout = FrameLayout(pix, n_nodes, ref, interp, cuda)
    slot = FrameSlot(layout, 12)
    slot.set_params(1e-6, 0.1)
    slot.load_image(frames[0])
    slot.set_u0(None)
    engine, desc = Engine(cuda, 1), descriptors_to_device([slot.desc], cuda)
    results = []
    for grid in (0, 1, 2, 7, 40):
        engine.solve(desc, 1, layout.kind, grid)
        torch.cuda.synchronize()
        results.append((slot.u_out.clone(), slot.hist.clone(), slot.info.clone()))
    for u, hist, info in results[1:]:
        assert torch.equal(u, results[0][0]) and torch.equal(info, results[0][2])
        assert torch.equal(hist.nan_to_num(7.0), results[0][1].nan_to_num(7.0))
    # one evaluation against the FP64 oracle, at the tolerance of the other gradient tests
    u = torch.as_tensor(np.random.default_rng(3).normal(0.0, 0.3, (n_nodes, 2)), dtype=torch.float32, device=cuda)
    J, g = engine.eval_objective(desc, u, layout.kind)
    oa = pixels.build_pixel_assets(np.asarray(mesh.nodes_xy), np.asarray(mesh.elements), side, side, assets.roi_mask)
    pb = objective.Problem.build(ref, frames[0], oa, interp)
    J64, g64 = objective.J_total_and_grad(u.cpu().numpy().astype(np.float64), pb, 0.1)
    assert abs(float(J) - J64) <= 1e-5 * J64
    assert np.abs(g.cpu().numpy() - g64).max() <= 1e-5 * np.abs(g64).max()


@pytest.mark.parametrize("slots", [2, 5])
def test_uneven_frames_finish_in_different_rounds(cuda, slots):
    """Several frames in one launch: the control steps of all frames, the rebuilt list, the last frame alone."""
    import d2ic_gb300 as d2
    from d2ic_gb300.engine import FrameLayout
    from d2ic_gb300.serving import solve_batch
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    work = []
    for i in range(slots):
        side = 72 + 40 * i
        ref, frames = speckle_sequence(side, side, [Translation(0.3, -0.2)], seed=90 + i, noise_seeds=[i, i + 50])
        mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 12, side - 12), 12)
        pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
        layout = FrameLayout(pix, mesh.nodes_xy.shape[0], ref, "cubic", cuda)
        work.append((layout, frames[0], None, d2.MeshDICConfig(max_iters=5 + 9 * i, tol=1e-6, reg_strength=0.1)))
    together = solve_batch(work)
    for w, got in zip(work, together):
        alone = solve_batch([w])[0]
        assert got[1] == alone[1] and np.array_equal(got[0], alone[0])
        assert np.array_equal(got[3], alone[3], equal_nan=True)


@pytest.mark.parametrize("side,element,move", [
    (1700, 6, 0.0),      # 36-pixel chunks, 32 per lane batch and more: about 33 chunks per warp
    (331, 7, 0.0),       # 49-pixel chunks: the second pixel of a pair is missing in lanes 17..31
    (300, 16, 0.0),      # full 256-pixel chunks
    (300, 16, 9.0),      # every stencil outside the tile placed before: the general path, then the packed one
    (95, 5, 3.0),        # 25-pixel chunks: no lane has a second pixel
])
def test_packed_pixels_and_lane_batches(cuda, side, element, move):
    """Chunks taken in batches of 32 and pixels two at a time: one evaluation against FP64 torch sums.

    The chunk boundaries and the last, partly filled batch are where a chunk or a pixel could be lost or
    counted twice; the tolerance is that of the other evaluations (FP32 residuals, sums of up to 2e6 terms)."""
    import d2ic_gb300 as d2
    from d2ic_gb300.engine import Engine, FrameLayout, FrameSlot, descriptors_to_device
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence_device
    ref, frames = speckle_sequence_device(side, side, [Translation(0.4 + move, -0.3 - move)], seed=5, noise_seeds=[5, 6])
    ref, frame = (np.asarray(x.cpu()) if torch.is_tensor(x) else np.asarray(x) for x in (ref, frames[0]))
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 24, side - 24), element)
    pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
    n_nodes = np.asarray(mesh.nodes_xy).shape[0]
    layout = FrameLayout(pix, n_nodes, ref, "cubic", cuda)
    slot = FrameSlot(layout, 4)
    slot.set_params(1e-6, 0.1)
    slot.load_image(frame)
    engine, desc = Engine(cuda, 1), descriptors_to_device([slot.desc], cuda)
    rng = np.random.default_rng(1)
    u = torch.as_tensor(rng.normal(0.0, 0.2, (n_nodes, 2)) + [move, -move], dtype=torch.float32, device=cuda)
    J, g = engine.eval_objective(desc, u, layout.kind)
    from oracle import objective, pixels
    oa = pixels.build_pixel_assets(np.asarray(mesh.nodes_xy), np.asarray(mesh.elements), side, side, assets.roi_mask)
    pb = objective.Problem.build(ref, frame, oa, "cubic")
    J64, g64 = objective.J_total_and_grad(u.cpu().numpy().astype(np.float64), pb, 0.1)
    assert abs(float(J) - J64) <= 1e-5 * J64
    assert np.abs(g.cpu().numpy() - g64).max() <= 1e-5 * np.abs(g64).max()


@pytest.mark.parametrize("frames,grid", [
    (2, 0), (16, 0), (17, 0),      # the most frames with their descriptors in shared memory, and one more
    (5, 9),                        # node groups on most warps of the grid
    (5, 3),                        # more groups than warps
    (16, 40),
])
def test_direct_rounds_of_several_frames(cuda, frames, grid):
    """Frames that hand over their own rules: pairs that finish in the same round, the list rebuilt down to one."""
    import d2ic_gb300 as d2
    from d2ic_gb300.engine import FrameLayout
    from d2ic_gb300.serving import solve_batch
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    work = []
    for i in range(frames):
        k = i // 2                                     # frames 2k and 2k + 1 are the same
        side = 64 + 24 * (k % 4)
        ref, images = speckle_sequence(side, side, [Translation(0.3, -0.2)], seed=40 + k, noise_seeds=[k, k + 50])
        mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 12, side - 12), 12 - 4 * (k % 2))
        pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
        layout = FrameLayout(pix, mesh.nodes_xy.shape[0], ref, "cubic", cuda)
        work.append((layout, images[0], None, d2.MeshDICConfig(max_iters=4 + 3 * k, tol=1e-6, reg_strength=0.1)))
    together = solve_batch(work, grid_blocks=grid)
    for w, got in zip(work, together):
        alone = solve_batch([w])[0]
        assert got[1] == alone[1] and np.array_equal(got[0], alone[0])
        assert np.array_equal(got[3], alone[3], equal_nan=True)


@pytest.mark.parametrize("n_nodes,k", [(1889, 4), (20_000, 1), (263_169, 4), (420_000, 3)])
def test_workspace_of_a_frame(n_nodes, k):
    """The workspace of a frame near the fixed scratch array's size: the buffers' sizes as the descriptor states them,
    double-float partials of the groups and supergroups, a counter for each, 256-byte aligned."""
    from d2ic_gb300 import _lib
    up = lambda x: (x + 255) // 256 * 256
    groups = (n_nodes + 31) // 32
    supers = (groups + 15) // 16
    want = up(56 * n_nodes) + up(16 * k * n_nodes) + up(40 * (groups + supers)) + up(4 * (groups + supers + 1)) + up(4 * n_nodes)
    assert _lib.load().d2ic_frame_workspace_bytes(n_nodes, n_nodes, k) == want

"""Evaluation tags of frames that have work in few blocks of the grid (GPU).

A block without a chunk or node group of a frame does not wait for the frame's control steps; its copy of the
frame's tag must not depend on when it reads it, or a later, shorter list that gives it work of the frame would
wait for records that never come.  Frames of 9 to 25 chunks finish one after the other, so that every list
change moves the rest to other blocks, in one launch and in slices that start at any evaluation; the results
are those of each frame alone.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,rounds", [
    (2, 0), (6, 0), (16, 0),
    (18, 0),          # a common release per round until 16 are left
    (66, 0),          # the list is read from memory until 64 are left
    (5, 1), (7, 3), (16, 4),
])
def test_list_changes_hand_few_chunks_on(cuda, frames, rounds):
    import d2ic_gb300 as d2
    from d2ic_gb300 import _lib
    from d2ic_gb300.engine import Engine, FrameLayout, FrameSlot, descriptors_to_device
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    layouts, images = [], []
    for k in range(3):
        side = 60 + 16 * k
        ref, moved = speckle_sequence(side, side, [Translation(0.3, -0.2)], seed=11 + k, noise_seeds=[k, k + 9])
        mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 12, side - 12), 16)
        pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
        layouts.append(FrameLayout(pix, mesh.nodes_xy.shape[0], ref, "cubic", cuda))
        images.append(moved[0])

    def slots_of(which):
        out = []
        for i in which:
            s = FrameSlot(layouts[i % 3], 3 + 2 * (i % 17))
            s.set_params(1e-6, 0.1)
            s.load_image(images[i % 3])
            s.set_u0(None)
            out.append(s)
        return out

    together = slots_of(range(frames))
    kind = layouts[0].kind
    engine, desc = Engine(cuda, frames), descriptors_to_device([s.desc for s in together], cuda)
    if rounds == 0:
        engine.solve(desc, frames, kind)
    else:
        engine.commands(frames).zero_()                # CMD_INIT
        for _ in range(1000):
            engine.run_slice(desc, frames, kind, rounds)
            torch.cuda.synchronize()
            if all(int(s.info[1]) != _lib.RUNNING for s in together):
                break
    torch.cuda.synchronize()
    alone = slots_of(range(min(frames, 51)))           # 3 images x 17 iteration limits
    for i, s in enumerate(alone):
        Engine(cuda, 1).solve(descriptors_to_device([s.desc], cuda), 1, kind)
    torch.cuda.synchronize()
    for i, s in enumerate(together):
        a = alone[i % 51]
        assert torch.equal(s.info, a.info) and torch.equal(s.u_out, a.u_out), i
        assert int(s.info[1]) in (_lib.OK, _lib.MAX_ITERS)

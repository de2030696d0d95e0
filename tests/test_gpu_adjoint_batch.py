"""Batched adjoint of the mixed term and transposed prefilter (GPU): the inner-product identity with the
forward maps over image sizes at the edges of the passes' blocks, batches, and displacements that leave
the chunk's tile or the image.

<A x, y> = <x, A^T y> in FP32 sums of up to 1e5 terms of either sign, compared in FP64: 2e-5 relative to
the norms.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,K", [(2, 3, 1), (17, 33, 2), (128, 130, 1), (129, 127, 3), (300, 4099, 1)])
def test_prefilter_transpose(cuda, H, W, K):
    from d2ic_gb300 import _lib
    from d2ic_gb300._lib import ptr
    from d2ic_gb300.engine import PAD, _pitch, prepare_coefficients
    g = torch.Generator(device=cuda).manual_seed(H * W)
    x = torch.randn((K, H, W), generator=g, device=cuda)
    cp = _pitch(W)
    y = torch.randn((K, H + 2 * PAD, cp), generator=g, device=cuda)
    tmp, xt = torch.empty((K, H, cp), device=cuda), torch.empty((K, H, W), device=cuda)
    _lib.call("d2ic_bspline_prefilter_T_batch", ptr(y), K, H, W, PAD, cp, ptr(tmp), ptr(xt), _lib.stream_handle())
    for k in range(K):
        c = prepare_coefficients(x[k].contiguous(), _lib.INTERP_CUBIC)[:, : W + 2 * PAD].double()
        yk = y[k, :, : W + 2 * PAD].double()
        a, b = float((c * yk).sum()), float((x[k].double() * xt[k].double()).sum())
        assert abs(a - b) <= 2e-5 * float(c.norm() * yk.norm())


@pytest.mark.parametrize("element,K,shift", [(12, 1, 0.0), (16, 5, 0.4), (32, 3, 0.0), (8, 33, 0.0), (16, 2, 60.0)])
def test_mixed_transpose(cuda, element, K, shift):
    import d2ic_gb300 as d2
    from d2ic_gb300.adjoint import ImplicitAdjoint
    from d2ic_gb300.engine import FrameLayout, FrameSlot
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence_device
    side = 150
    ref, frames = speckle_sequence_device(side, side, [Translation(0.3, -0.4)], seed=5, noise_seeds=[1, 2], device=cuda,
                                          u8=False)
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 8, side - 8), element)
    pix = d2.build_pixel_assets(mesh, ref.cpu().numpy(), 1.0, assets.roi_mask)
    layout = FrameLayout(pix, mesh.nodes_xy.shape[0], ref, "cubic", cuda)
    slot = FrameSlot(layout, 1)
    slot.load_image(frames[0])
    rng = np.random.default_rng(element)
    # rough displacements: stencil corners shared by pixels of a step, boxes wider than the tile for some
    # chunks, and (shift) stencils beyond the image's border
    u = torch.as_tensor(rng.normal(0, 3.0, (layout.n_nodes, 2)) + shift, dtype=torch.float32, device=cuda)
    adj = ImplicitAdjoint(slot, u, 0.1)
    g = torch.Generator(device=cuda).manual_seed(K)
    dI = torch.randn((K, side, side), generator=g, device=cuda)
    lam = torch.randn((layout.n_nodes, 2, K), generator=g, device=cuda)
    fwd, bwd = adj.mixed(dI), adj.mixed_T(lam)
    for k in range(K):
        a = float((fwd[:, :, k] * lam[:, :, k].double()).sum())
        b = float((dI[k].double() * bwd[k].double()).sum())
        scale = float(dI[k].double().norm() * bwd[k].double().norm())
        assert abs(a - b) <= 2e-5 * scale


@pytest.mark.parametrize("element,K,spread", [(8, 1, 0.2), (13, 9, 0.2), (16, 33, 0.2), (24, 17, 0.2), (16, 40, 8.0),
                                              (12, 16, 0.2)])
def test_mixed_batch_matches_single_images_and_fp64(cuda, element, K, spread):
    """Image counts around the images a warp and a block take at a time, coefficients that cannot be copied 16 bytes
    at a time, windows that do not fit: the same bits as one image per call, and the FP64 oracle."""
    import d2ic_gb300 as d2
    from d2ic_gb300 import _lib
    from d2ic_gb300._lib import ptr
    from d2ic_gb300.engine import PAD, FrameLayout, FrameSlot, descriptors_to_device, prepare_coefficients
    from d2ic_gb300.synthetic import Translation, rect_mask, speckle_sequence
    from oracle import adjoint as oadj
    from oracle import objective, pixels
    side = 90
    ref, frames = speckle_sequence(side, side, [Translation(0.3, -0.4)], seed=5, noise_seeds=[1, 2])
    mesh, assets = d2.mask_to_mesh_assets(rect_mask(side, side, side - 8, side - 8), element)
    pix = d2.build_pixel_assets(mesh, ref, 1.0, assets.roi_mask)
    L = FrameLayout(pix, mesh.nodes_xy.shape[0], ref, "cubic", cuda)
    slot = FrameSlot(L, 1)
    slot.load_image(frames[0])
    desc = descriptors_to_device([slot.desc], cuda)
    rng = np.random.default_rng(element)
    u = torch.as_tensor(rng.normal(0, spread, (L.n_nodes, 2)), dtype=torch.float32, device=cuda)
    dI = rng.normal(0, 1, (K, side, side)).astype(np.float32)
    co = torch.stack([prepare_coefficients(torch.as_tensor(x, device=cuda), _lib.INTERP_CUBIC) for x in dI])
    size = (L.H + 2 * PAD) * L.cpitch
    slots = torch.zeros((K, L.node_chunk_k * L.n_nodes, 2), device=cuda)
    outs = []
    for offset in (0, 1):                              # 1: rows start between 16-byte boundaries
        flat = torch.zeros(K * (size + offset) + 4, device=cuda)
        for k in range(K):
            flat[offset + k * (size + offset):][:size] = co[k].reshape(-1)
        out = torch.zeros((L.n_nodes, 2, K), device=cuda)
        _lib.call("d2ic_mixed_term_batch", ptr(desc), L.n_chunks, L.n_nodes, L.node_chunk_k, ptr(u),
                  flat.data_ptr() + 4 * offset, K, size + offset, 1.0, ptr(slots), ptr(out), K, 0, _lib.stream_handle())
        outs.append(out)
    one = torch.zeros((L.n_nodes, 2, K), device=cuda)
    for k in range(K):
        _lib.call("d2ic_mixed_term", ptr(desc), L.n_chunks, L.n_nodes, ptr(u), ptr(co[k]), 1.0, ptr(slots), ptr(one), K, k,
                  _lib.stream_handle())
    assert torch.equal(outs[0], one) and torch.equal(outs[1], one)
    oa = pixels.build_pixel_assets(np.asarray(mesh.nodes_xy), np.asarray(mesh.elements), side, side, assets.roi_mask)
    pb = objective.Problem.build(ref, frames[0], oa, "cubic")
    want = np.asarray(oadj.mixed_term(u.cpu().numpy().astype(np.float64), pb, dI[0].astype(np.float64))).reshape(-1, 2)
    got = one[:, :, 0].cpu().numpy().astype(np.float64) / L.n_pix
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()

"""ZNCC scores of windows whose mean lies far from the mean of their search patch (GPU), against the FP64 oracle.

Running sums over the centred patch lose digits with (window mean - patch mean)^2 / variance; windows beyond
the line where that costs more than the two-pass form's serial FP32 sums are scored in two passes.  The bound
is that form's: its largest error among 2,000 simulated windows of correlation 0.99, 0.6, 0.7, 1.1 and 1.3e-6 at win 9,
11, 15 and 21, doubled.  (Running sums up to 8 standard deviations have 2.3e-6 and 2.5e-6 at win 9 and 11.)
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("win,search,tol", [(7, 12, 1.2e-6), (9, 12, 1.2e-6), (11, 8, 1.4e-6), (11, 14, 1.4e-6),
                                            (15, 12, 2.2e-6), (21, 6, 2.6e-6)])
@pytest.mark.parametrize("sd", [10.0, 0.05])
def test_windows_off_the_patch_mean(cuda, win, search, tol, sd):
    from d2ic_gb300.solver_translation_zncc import match_centers_device
    from oracle.init_motion import match_centers
    rng = np.random.default_rng(win * 100 + search)
    tile, n = win + 2 * search + 16, 20
    edge = tile // 2                                       # dark columns left of it, bright ones right
    at = edge + win // 2 + 4
    # the dark part of the patch around a centre, and the brightness that puts its windows q deviations off
    left = search - 4
    dark = left / (win + 2 * search)
    q = rng.uniform(0.0, 9.0, (n, n))
    ref = np.kron(q * sd / dark, np.ones((tile, tile)))
    ref[:, np.arange(n * tile) % tile < edge] = 0.0
    ref = (ref + sd * rng.standard_normal(ref.shape)).astype(np.float32)
    img = (np.roll(ref, (2, 1), (0, 1)) + 0.05 * sd * rng.standard_normal(ref.shape)).astype(np.float32)
    y, x = np.mgrid[:n, :n]
    centres = np.stack([x.ravel() * tile + at, y.ravel() * tile + tile // 2], axis=1).astype(np.float32)
    u, s = match_centers_device(centres, torch.as_tensor(ref, device=cuda), torch.as_tensor(img, device=cuda), win, search,
                                cuda)
    u, s = u.cpu().numpy(), s.cpu().numpy()
    u64, s64 = match_centers(centres, ref, img, win, search)
    ok = ~np.isnan(s64)
    assert np.array_equal(ok, ~np.isnan(s)) and ok.sum() >= 200
    assert np.array_equal(u[ok], u64[ok]) and (u64[ok] == [1, 2]).all()
    assert np.abs(s[ok] - s64[ok]).max() <= tol, np.abs(s[ok] - s64[ok]).max()


def test_few_and_many_windows_of_a_block(cuda):
    """A weakly textured field with one to many bright spots: the windows left to the two-pass form are none, a few
    (scored by a warp each) or most of a block's."""
    from d2ic_gb300.solver_translation_zncc import match_centers_device
    from oracle.init_motion import match_centers
    rng = np.random.default_rng(3)
    ref = rng.normal(0, 1.0, (400, 400)).astype(np.float32)
    for k, x in enumerate(range(40, 400, 40)):
        for _ in range(k * k):
            ref[rng.integers(0, 400), x + rng.integers(-18, 19)] += 200.0
    img = (np.roll(ref, (1, -2), (0, 1)) + rng.normal(0, 0.05, ref.shape)).astype(np.float32)
    centres = np.stack([v.ravel() for v in np.meshgrid(np.arange(30, 371, 20), np.arange(30, 371, 20))], 1).astype(np.float32)
    for win, search in ((11, 9), (21, 8), (17, 3)):
        u, s = match_centers_device(centres, torch.as_tensor(ref, device=cuda), torch.as_tensor(img, device=cuda), win,
                                    search, cuda)
        u64, s64 = match_centers(centres, ref, img, win, search)
        assert np.array_equal(u.cpu().numpy(), u64)
        assert np.abs(s.cpu().numpy() - s64).max() <= 2.6e-6

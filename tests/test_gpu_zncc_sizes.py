"""ZNCC search over its range of windows and search distances (GPU) against the FP64 oracle.

Sizes sit at the edges of the register blocking (rows in pairs, 5 to 7 columns of offsets per thread,
windows that are not a multiple of that) and on both sides of the line to the wide form.  A score is a
mean of at most 61^2 products of values of unit variance, summed in FP32: 5e-6 covers the rounding.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SCORE_TOL = 5e-6


def _match(ref, img, centres, win, search, device):
    from d2ic_gb300.solver_translation_zncc import match_centers_device
    u, s = match_centers_device(centres, torch.as_tensor(ref, device=device), torch.as_tensor(img, device=device), win,
                                search, device)
    return u.cpu().numpy(), s.cpu().numpy()


@pytest.mark.parametrize("win,search", [(1, 0), (3, 1), (5, 3), (7, 2), (17, 8), (21, 5), (15, 14), (41, 24), (9, 34),
                                        (9, 40), (61, 12)])
def test_scores_and_shifts_match_the_oracle(cuda, win, search):
    from oracle.init_motion import match_centers
    rng = np.random.default_rng(win * 100 + search)
    size = win + 2 * search + 40
    ref = (120 + 60 * rng.standard_normal((size, size + 6))).astype(np.float32)
    img = np.roll(ref, (min(search, 2), -min(search, 1)), (0, 1)) + rng.normal(0, 3, ref.shape).astype(np.float32)
    centres = np.stack([rng.uniform(0, size + 6, 40), rng.uniform(0, size, 40)], axis=1).astype(np.float32)
    u, s = _match(ref, img, centres, win, search, cuda)
    u64, s64 = match_centers(centres, ref, img, win, search)
    assert np.array_equal(np.isnan(s), np.isnan(s64))
    ok = ~np.isnan(s64)
    assert ok.any()
    if win > 1:
        assert np.array_equal(u, u64)
        assert np.abs(s[ok] - s64[ok]).max() <= SCORE_TOL


def test_flat_bright_and_missing_pixels(cuda):
    """Windows with almost no variance beside bright ones, a constant patch, and pixels that are not numbers."""
    from oracle.init_motion import match_centers
    rng = np.random.default_rng(5)
    ref = rng.normal(0, 1.0, (120, 120)).astype(np.float32) + 20
    ref[:, 60:] += 4000 * (rng.random((120, 60)) > 0.5)        # windows of very different mean and variance
    img = np.roll(ref, 2, 0)
    centres = np.array([[40, 60], [55, 60], [80, 60], [50.5, 40.5]], np.float32)
    u, s = _match(ref, img, centres, 11, 9, cuda)
    u64, s64 = match_centers(centres, ref, img, 11, 9)
    assert np.array_equal(u, u64) and np.abs(s - s64).max() <= SCORE_TOL
    flat = np.full((120, 120), 37.0, np.float32)
    u, s = _match(flat, flat, centres, 11, 9, cuda)
    assert np.array_equal(u, np.full((4, 2), -9.0)) and np.array_equal(s, np.zeros(4))
    # a pixel that is not a number only spoils the windows that hold it: the search around it goes through
    # the two-pass form, whose result for a clean best window beside it is the oracle's
    img2 = img.copy()
    img2[60, 100] = np.nan
    far = np.array([[30, 60], [40, 40]], np.float32)
    assert np.array_equal(_match(ref, img2, far, 11, 9, cuda)[0], match_centers(far, ref, img2, 11, 9)[0])


@pytest.mark.parametrize("win,search", [(11, 6), (11, 7), (17, 8), (21, 5), (15, 9), (9, 20), (31, 3)])
def test_many_centres(cuda, win, search):
    """More centres than SMs: the blocked form at its small sizes and the line to the wide one."""
    from oracle.init_motion import match_centers
    rng = np.random.default_rng(win + search)
    size = 150
    ref = (120 + 60 * rng.standard_normal((size, size + 3))).astype(np.float32)
    img = np.roll(ref, (2, -1), (0, 1)) + rng.normal(0, 3, ref.shape).astype(np.float32)
    centres = np.stack([rng.uniform(0, size + 3, 200), rng.uniform(0, size, 200)], axis=1).astype(np.float32)
    u, s = _match(ref, img, centres, win, search, cuda)
    u64, s64 = match_centers(centres, ref, img, win, search)
    assert np.array_equal(np.isnan(s), np.isnan(s64))
    ok = ~np.isnan(s64)
    assert ok.any() and np.array_equal(u, u64) and np.abs(s[ok] - s64[ok]).max() <= SCORE_TOL

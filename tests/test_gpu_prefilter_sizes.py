"""B-spline prefilter at the edges of its blocks (GPU): 128 columns, 32, 64 or 128 rows per block, single rows
and columns, 8-bit pixels and batches, against the same sums in FP64."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fir(x, axis, pad):
    h = np.array([np.sqrt(3.0) * (np.sqrt(3.0) - 2.0) ** abs(k) for k in range(-16, 17)])
    n = x.shape[axis]
    at = np.arange(-pad, n + pad)
    return sum(h[k + 16] * np.take(x, np.clip(at + k, 0, n - 1), axis) for k in range(-16, 17))


@pytest.mark.parametrize("n,H,W,pad,u8", [
    (1, 1, 1, 16, False), (1, 5, 97, 16, True), (1, 33, 96, 16, False), (1, 300, 95, 17, False),
    (3, 65, 225, 16, False), (1, 512, 640, 16, True), (7, 700, 333, 20, False), (1, 1500, 2050, 16, False),
])
def test_prefilter_against_fp64(cuda, n, H, W, pad, u8):
    from d2ic_gb300 import _lib
    from d2ic_gb300._lib import ptr
    rng = np.random.default_rng(H + W)
    img = rng.integers(0, 256, (n, H, W)).astype(np.uint8 if u8 else np.float32)
    cp = W + 2 * pad + 3                                   # rows that are not aligned
    x = torch.as_tensor(img, device=cuda)
    tmp = torch.empty((n, H, cp), dtype=torch.float32, device=cuda)
    out = torch.full((n, H + 2 * pad, cp), 7.0, dtype=torch.float32, device=cuda)
    if u8:
        _lib.call("d2ic_bspline_prefilter_u8", ptr(x), H, W, pad, cp, ptr(tmp), ptr(out), _lib.stream_handle())
    else:
        _lib.call("d2ic_bspline_prefilter_batch", ptr(x), n, H, W, pad, cp, ptr(tmp), ptr(out), _lib.stream_handle())
    got = out.cpu().numpy()
    assert (got[:, :, W + 2 * pad:] == 7.0).all()          # nothing past a row's end
    ref = _fir(_fir(img.astype(np.float64), 2, pad), 1, pad)
    # 33 rounded sums per pass, |h| sums to 3 per pass
    assert np.abs(got[:, :, :W + 2 * pad] - ref).max() <= 66 * 6e-8 * 9 * 255

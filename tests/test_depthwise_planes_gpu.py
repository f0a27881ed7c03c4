"""Depthwise layers of small planes at the plane counts where the number of planes per CTA changes, against 64-bit sums.

Tolerance: a sum of K fp32 products and a bias is off by at most (K + 2) 2^-24 sum|terms|."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT, _ref

from test_plane_sums_gpu import params


def windows(x, w, k, stride):
    pad = (k - 1) // 2
    x = np.pad(x, ((0, 0), (0, 0), (pad, pad), (pad, pad)))
    v = np.lib.stride_tricks.sliding_window_view(x, (k, k), (2, 3))[:, :, ::stride, ::stride]
    return np.einsum("nchwij,cij->nchw", v, w[:, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("k,stride", [(3, 1), (5, 1), (3, 2), (5, 2)])
@pytest.mark.parametrize("n,c,h", [(1, 4, 7), (1, 12, 7), (1, 588, 7), (1, 592, 14), (1, 596, 14), (1, 1172, 7), (2, 600, 7), (3, 796, 5), (1, 240, 28), (7, 388, 14)])
def test_small_planes(n, c, h, k, stride):
    rng = np.random.default_rng(n * c + h)
    x, w, b = rng.standard_normal((n, c, h, h)).astype(np.float32), rng.standard_normal((c, 1, k, k)).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    dx, dw, db = DT.from_numpy(x), DT.from_numpy(w), DT.from_numpy(b)
    o = (h - 1) // stride + 1
    y = DT.from_numpy(np.full((n, c, o, o), np.nan, np.float32))
    p = params(c, k, stride, cabi.ACT_NONE)
    cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(dw), _ref(db), _ref(y), ctypes.byref(p), None))
    cabi.check_device()
    x, w, b = x.astype(np.float64), w.astype(np.float64), b.astype(np.float64)[:, None, None]
    off = np.abs(y.numpy() - (windows(x, w, k, stride) + b))
    assert (off <= (k * k + 2) * 2.0 ** -24 * (windows(np.abs(x), np.abs(w), k, stride) + np.abs(b))).all()

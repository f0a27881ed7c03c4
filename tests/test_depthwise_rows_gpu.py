"""1-D depthwise layers over channel-innermost operands, at the edges of the run of positions a thread takes.

Tolerance: K fp32 products, a bias: (K + 2) 2^-24 sum|terms|."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import ConvParams, DeviceTensor as DT, _ref


@pytest.mark.gpu
@pytest.mark.parametrize("k", [3, 5, 7, 9, 4])
@pytest.mark.parametrize("n,c,length,out", [(1, 4, 1, 1), (2, 256, 7, 7), (1, 260, 8, 8), (3, 12, 9, 9), (1, 768, 130, 130), (2, 20, 33, 29), (1, 8, 6, 14), (5, 1028, 16, 16)])
@pytest.mark.parametrize("packed", [True, False])
def test_runs(n, c, length, out, k, packed):
    rng = np.random.default_rng(c + length + k)
    x, w, b = rng.standard_normal((n, length, c)).astype(np.float32), rng.standard_normal((c, 1, k)).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    w[0, 0, 0] = np.inf if length < 8 else w[0, 0, 0]     # a tap over the padding is left out, not multiplied by zero
    pad = (out - length + k - 1 + 1) // 2 if out >= length - k + 1 else 0
    dx, dw, db = DT.from_numpy(x), DT.from_numpy(w, None if packed else [1, 2, 0]), DT.from_numpy(b)
    y = DT.from_numpy(np.full((n, out + 1, c + 4), np.nan, np.float32))
    p = ConvParams()
    p.pads_begin[0], p.strides[0], p.dilations[0], p.group, p.act, p.precision = pad, 1, 1, c, cabi.ACT_NONE, cabi.GEMM_AUTO
    vx = dx.view((n, c, length), [length * c, 1, c], 0)
    vy = y.view((n, c, out), [(out + 1) * (c + 4), 1, c + 4], 0)
    cabi.check(cabi.lib().fml_conv(_ref(vx), _ref(dw), _ref(db), _ref(vy), ctypes.byref(p), None))
    cabi.check_device()
    got = y.numpy()
    assert np.isnan(got[:, out]).all() and np.isnan(got[:, :, c:]).all()
    ref, total = np.zeros((n, out, c)) + b, np.zeros((n, out, c)) + np.abs(b)
    for o in range(out):
        for j in range(k):
            i = o - pad + j
            if 0 <= i < length:
                t = x[:, i].astype(np.float64) * w[:, 0, j]
                ref[:, o] += t
                total[:, o] += np.abs(t)
    got, sane = got[:, :out, :c], np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), sane) and (np.abs(got[sane] - ref[sane]) <= (k + 2) * 2.0 ** -24 * total[sane]).all()

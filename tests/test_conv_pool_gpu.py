"""A convolution that pools its result: the same numbers as the convolution with the same tiles, then the 2 x 2 maximum.

Exact: scaling by powers of two, adding the bias and ReLU keep order, so the maximum may come first."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi, models
from fluidml_b200.cabi import ConvParams, DeviceTensor as DT, _ref
from fluidml_b200.executor import Executor

from test_conv_pointwise_gpu import Host


def params(pad, act=cabi.ACT_RELU, tiles=(0, 0, 0, 0)):
    p = ConvParams()
    for i in range(2):
        p.pads_begin[i], p.strides[i], p.dilations[i] = pad, 1, 1
    p.group, p.act, p.precision = 1, act, cabi.GEMM_AUTO
    p.tile_n, p.strips, p.split_k, p.ctas_per_sm = tiles
    return p


def uses(x, w, y, p, scaled=0):
    n = ctypes.c_int()
    cabi.check(cabi.lib().fml_conv_uses_packed(_ref(x), _ref(w), _ref(y), ctypes.byref(p), scaled, ctypes.byref(n)))
    return n.value


@pytest.mark.gpu
@pytest.mark.parametrize("n,ic,oc,h,w,k,pad", [
    (2, 32, 64, 24, 40, 3, 1), (1, 48, 36, 18, 20, 3, 1), (1, 64, 128, 16, 8, 3, 1), (1, 40, 32, 22, 12, 5, 2), (3, 64, 16, 18, 36, 3, 0),  # boxes
    (2, 256, 96, 14, 14, 3, 1), (1, 96, 260, 10, 10, 3, 1), (1, 512, 512, 14, 14, 3, 1),                                                  # flattened rows
    (2, 3, 64, 32, 32, 3, 1), (1, 6, 36, 18, 36, 3, 1),                                                                                   # channel x tap
])
@pytest.mark.parametrize("tiles", [(0, 0, 0, 0), (32, 1, 1, 2), (64, 2, 1, 1), (64, 1, 8, 2), (32, 2, 4, 1), (64, 2, 8, 1), (128, 2, 2, 1)])
@pytest.mark.parametrize("odd", [False, True])
def test_the_maximum_of_the_convolution(n, ic, oc, h, w, k, pad, tiles, odd):
    rng = np.random.default_rng(ic + oc + h)
    x, wt, b = rng.standard_normal((n, ic, h, w)).astype(np.float32), rng.standard_normal((oc, ic, k, k)).astype(np.float32), rng.standard_normal(oc).astype(np.float32)
    if odd:  # values that are no numbers, and columns of very different size
        x[0, 0, 3, 5], x[0, ic - 1, 8, 2], x[0, ic // 2, 9, 7] = np.nan, np.inf, -np.inf
        wt *= np.exp2(rng.integers(-40, 40, (oc, 1, 1, 1))).astype(np.float32)
        b[: oc // 2] = -3
    oh, ow = h + 2 * pad - k + 1, w + 2 * pad - k + 1
    dx, dw, db = DT.from_numpy(x), DT.from_numpy(wt, [3, 2, 0, 1]), DT.from_numpy(b)
    full, y = DT((n, oc, oh, ow), np.float32), DT.from_numpy(np.full((n, oc, oh // 2, ow // 2), -1, np.float32))
    packed = cabi.conv_pack(dw)
    p = params(pad, tiles=tiles)
    p.w_packed = packed.ptr
    cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(dw), _ref(db), _ref(full), ctypes.byref(p), None))
    p.max_pool = 1
    assert uses(dx, dw, y, p)
    cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(dw), _ref(db), _ref(y), ctypes.byref(p), None))
    cabi.check_device()
    f = full.numpy()
    ref = f.reshape(n, oc, oh // 2, 2, ow // 2, 2).max((3, 5))
    assert not np.isnan(f).any() and np.array_equal(y.numpy(), ref)


def test_where_nothing_is_pooled():
    x, w, y, last = Host((1, 32, 32, 32)), Host((64, 32, 3, 3), [3, 2, 0, 1]), Host((1, 64, 16, 16)), Host((1, 64, 16, 16), [0, 3, 1, 2])
    for act, k, want in ((cabi.ACT_RELU, 3, 1), (cabi.ACT_NONE, 3, 0), (cabi.ACT_SILU, 3, 0), (cabi.ACT_RELU, 1, 0)):
        p = params(k // 2, act)
        p.max_pool = 1
        w = Host((64, 32, k, k), [3, 2, 0, 1])
        assert uses(x, w, y, p) == want and uses(x, w, last, p) == want and uses(x, w, y, p, 1) == 0
        p.precision = cabi.GEMM_FP32
        assert uses(x, w, y, p) == 0
        assert cabi.lib().fml_conv(_ref(x), _ref(w), None, _ref(y), ctypes.byref(p), None) != 0


def pools_left(side=32, act=True, pool=(2, 2), read_twice=False):
    g = models.GraphBuilder("pools")
    x = g.input("x", 1, (1, 32, side, side))
    y = g.conv(x, g.const("w", np.ones((64, 32, 3, 3), np.float32)), pads=[1, 1, 1, 1])
    y = g.relu(y) if act else y
    z = g.maxpool(y, list(pool), [2, 2])
    g.output(g.sqrt(z, "out"))
    if read_twice:
        g.output(g.neg(y, "more"))
    st = Executor.make_dp_greedy("t").plan(g.finish().to_bytes())
    return sum(n["kind"] == "MaxPoolWithoutPadding" for n in st["sequence"])


def test_the_plan_folds_what_it_may():
    assert pools_left() == 0
    assert pools_left(side=13) == 1          # the convolution's last row and column belong to no window
    assert pools_left(act=False) == 1
    assert pools_left(pool=(3, 3)) == 1
    assert pools_left(read_twice=True) == 1


def test_the_plan_folds_the_pools_of_vgg16():
    st = Executor.make_dp_greedy("t").plan(models.build_vgg16().to_bytes())
    assert not [n for n in st["sequence"] if n["kind"] == "MaxPoolWithoutPadding"]

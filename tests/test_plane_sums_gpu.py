"""The sums of its planes that a depthwise convolution leaves, and the gate that starts from them.

Tolerance: a sum of K fp32 terms, in any order, is off by at most K 2^-24 sum|terms|; carried through the gate's layers."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from fluidml_b200 import cabi, models
from fluidml_b200.cabi import ConvParams, DeviceTensor as DT, _ref
from fluidml_b200.executor import Executor

from test_conv_pointwise_gpu import Host


def params(c, k, stride, act):
    p = ConvParams()
    for i in range(2):
        p.pads_begin[i], p.strides[i], p.dilations[i] = (k - 1) // 2, stride, 1
    p.group, p.act, p.precision = c, act, cabi.GEMM_AUTO
    return p


def parts_of(x, w, y, p):
    n = ctypes.c_int()
    cabi.check(cabi.lib().fml_conv_plane_sum_parts(_ref(x), _ref(w), _ref(y), ctypes.byref(p), ctypes.byref(n)))
    return n.value


def alone(code):
    """What a process of its own, without a device, has to say about `code`: nothing when it ends well."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", code], cwd=root, env={**os.environ, "CUDA_VISIBLE_DEVICES": "", "PYTHONPATH": root}, capture_output=True, text=True)
    return "" if done.returncode == 0 else f"{done.returncode}: {done.stderr}"


@pytest.mark.gpu
@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("n,c,h,w", [(1, 32, 112, 112), (2, 16, 56, 56), (1, 8, 18, 20), (3, 12, 33, 64), (1, 480, 14, 14), (3, 20, 7, 7), (1, 4, 4, 4), (2, 6, 15, 13),
                                     (1, 3, 200, 240), (5, 40, 16, 16)])
def test_sums_of_the_planes(k, stride, n, c, h, w):
    rng = np.random.default_rng(h * w + c)
    act = cabi.ACT_SILU if c % 3 else cabi.ACT_NONE
    x, wt, b = rng.standard_normal((n, c, h, w)).astype(np.float32), rng.standard_normal((c, 1, k, k)).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    dx, dw, db = DT.from_numpy(x), DT.from_numpy(wt), DT.from_numpy(b)
    y = DT((n, c, (h - 1) // stride + 1, (w - 1) // stride + 1), np.float32)
    p = params(c, k, stride, act)
    parts = parts_of(dx, dw, y, p)
    if parts == 0:
        assert w < 16 or w % 4  # only planes that the narrow kernel does not take either
        return
    sums = DT.from_numpy(np.full((n * c + 1, parts), np.nan, np.float32))
    p.plane_sums = sums.c().data
    cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(dw), _ref(db), _ref(y), ctypes.byref(p), None))
    cabi.check_device()
    got, out = sums.numpy(), y.numpy().reshape(n * c, -1).astype(np.float64)
    assert np.isnan(got[n * c]).all() and np.isfinite(got[:n * c]).all()
    bound = out.shape[1] * 2.0 ** -24 * np.abs(out).sum(1) + 1e-30
    assert (np.abs(got[:n * c].astype(np.float64).sum(1) - out.sum(1)) <= bound).all()
    ref = DT(y.shape, np.float32)  # and the result is the one without sums
    p.plane_sums = None
    cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(dw), _ref(db), _ref(ref), ctypes.byref(p), None))
    assert np.array_equal(ref.numpy(), y.numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("n,c,cr,parts", [(1, 32, 8, 7), (2, 96, 4, 1), (1, 1152, 48, 1), (3, 7, 2, 3), (1, 2, 1, 1), (64, 240, 10, 2), (19, 4096, 512, 1), (130, 33, 20, 5)])
def test_the_gate_from_sums(n, c, cr, parts):
    rng = np.random.default_rng(c)
    sums = rng.standard_normal((n, c, parts)).astype(np.float32) * 50
    w1, w2 = rng.standard_normal((cr, c, 1, 1)).astype(np.float32) * 0.1, rng.standard_normal((c, cr, 1, 1)).astype(np.float32)
    b1, b2 = rng.standard_normal(cr).astype(np.float32), rng.standard_normal(c).astype(np.float32)
    gate = DT((n, c, 1, 1), np.float32)
    ds, d1, db1, d2, db2 = (DT.from_numpy(t) for t in (sums, w1, b1, w2, b2))
    cabi.check(cabi.lib().fml_squeeze_excite_gate_from_sums(_ref(ds), ctypes.c_int64(196), _ref(d1), _ref(db1), _ref(d2), _ref(db2), cabi.ACT_SILU,
                                                            cabi.ACT_SIGMOID, _ref(gate), None))
    cabi.check_device()
    m, v1, v2 = sums.astype(np.float64).sum(2) / 196, w1[:, :, 0, 0].T.astype(np.float64), w2[:, :, 0, 0].T.astype(np.float64)
    m_off = (parts + 1) * 2.0 ** -24 * np.abs(sums).sum(2) / 196
    h = m @ v1 + b1
    h_off = (c + 2) * 2.0 ** -24 * (np.abs(m) @ np.abs(v1) + np.abs(b1)) + m_off @ np.abs(v1)
    a = h / (1 + np.exp(-h))
    a_off = 1.1 * h_off + 4 * 2.0 ** -24 * np.abs(a)                      # SiLU's slope is below 1.1
    g = a @ v2 + b2
    g_off = (cr + 2) * 2.0 ** -24 * (np.abs(a) @ np.abs(v2) + np.abs(b2)) + a_off @ np.abs(v2)
    off = np.abs(gate.numpy()[:, :, 0, 0] - 1 / (1 + np.exp(-g)))
    assert (off <= g_off / 4 + 4 * 2.0 ** -24).all()                      # the sigmoid's slope is at most 1 / 4


def test_where_there_are_no_sums():
    p = params(8, 3, 1, cabi.ACT_NONE)
    x, w, y = Host((1, 8, 32, 32)), Host((8, 1, 3, 3)), Host((1, 8, 32, 32))
    assert parts_of(x, w, y, p) > 0
    p.dilations[0] = 2
    assert parts_of(x, w, y, p) == 0
    p = params(1, 3, 1, cabi.ACT_NONE)
    assert parts_of(x, Host((8, 8, 3, 3)), y, p) == 0                    # not depthwise
    p = params(8, 7, 1, cabi.ACT_NONE)
    assert parts_of(x, Host((8, 1, 7, 7)), y, p) == 0                    # another kernel's window
    last = [0, 3, 1, 2]
    p = params(8, 3, 1, cabi.ACT_NONE)
    assert parts_of(Host((1, 8, 32, 32), last), w, Host((1, 8, 32, 32), last), p) == 0  # channels innermost


@pytest.mark.parametrize("x,y", [((1, 8, 32, 32), (1, 8, 0, 32)), ((1, 8, 7, 7), (1, 8, 7, 0)), ((1, 8, 0, 32), (1, 8, 0, 32)), ((0, 8, 32, 32), (0, 8, 32, 32)),
                                 ((0, 8, 7, 7), (0, 8, 7, 7))])
def test_empty_planes_have_no_sums(x, y):
    code = f"""if True:
        import sys
        sys.path[:0] = ["tests"]
        from test_plane_sums_gpu import Host, params, parts_of
        assert parts_of(Host({x}), Host((8, 1, 3, 3)), Host({y}), params(8, 3, 1, 0)) == 0
    """
    assert alone(code) == ""  # a process of its own: a division by zero would end this one


def test_a_layer_that_cannot_leave_its_sums_is_an_error():
    """Without a device there is no status word: the layer must not go on to a kernel that ignores the sums."""
    code = """if True:
        import ctypes, sys
        sys.path[:0] = ["tests"]
        from test_plane_sums_gpu import Host, cabi, params
        for size in (32, 7):   # either of the kernels that leave sums
            x, w, y, sums = Host((1, 8, size, size)), Host((8, 1, 3, 3)), Host((1, 8, size, size)), Host((8, 1))
            p = params(8, 3, 1, cabi.ACT_NONE)
            p.plane_sums = sums.c().data
            try:
                cabi.check(cabi.lib().fml_conv(ctypes.byref(x.c()), ctypes.byref(w.c()), None, ctypes.byref(y.c()), ctypes.byref(p), None))
            except cabi.FmlError as e:
                assert "plane sums" in str(e), e
            else:
                raise SystemExit("no error")
    """
    assert alone(code) == ""


def test_the_plan_gives_the_sums_a_place():
    st = Executor.make_dp_greedy("t").plan(models.build_efficientnet_b0(batch=1, image=64, std=0.16).to_bytes())
    gates = [n for n in st["sequence"] if n["kind"] == "SqueezeExciteGate"]
    assert len(gates) == 16 and all(any(i.endswith("_plane_sums") for i in n["inputs"]) for n in gates)

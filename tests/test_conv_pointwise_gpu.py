"""The fp32 FMA kernel of pointwise convolutions against fp64: edges of its 32-channel x 32-pixel tiles, every split of k,
gates, residuals, planes whose rows are not 16-byte aligned, and operands inside wider buffers.

Tolerance: a sum of K products in fp32, in any order, is off by at most K 2^-24 sum|w x|, one rounding each for the gate
and the bias; the activations' slopes are at most 1.1 and their own error a few ulp."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi, models
from fluidml_b200.cabi import ConvParams, DeviceTensor as DT, _ref
from fluidml_b200.executor import Executor

ACTS = {cabi.ACT_NONE: lambda y: y, cabi.ACT_SILU: lambda y: y / (1 + np.exp(-y)), cabi.ACT_RELU: lambda y: np.maximum(y, 0)}


def params(act, wk, split):
    p = ConvParams()
    for i in range(2):
        p.strides[i] = p.dilations[i] = 1
    p.group, p.act, p.precision, p.pointwise_fma, p.tile_n, p.split_k = 1, act, cabi.GEMM_AUTO, 1, wk, split
    return p


def run(x, w, bias, gate, res, act, wk=0, split=0, pad=0):
    """y inside a buffer with `pad` planes more per image, which have to keep what they hold."""
    n, oc, (h, wd) = x.shape[0], w.shape[0], x.shape[2:]
    buf = DT.from_numpy(np.full((n, oc + pad, h, wd), 7.0, np.float32))
    view = lambda t: t.view((n, oc, h, wd), [(oc + pad) * h * wd, h * wd, wd, 1], 0)
    y = view(buf)
    dw, dx, db = DT.from_numpy(w, [3, 2, 0, 1]), DT.from_numpy(x), DT.from_numpy(bias)
    dg = DT.from_numpy(gate) if gate is not None else None
    p = params(act, wk, split)
    if res is not None:
        wide = np.zeros((n, oc + pad, h, wd), np.float32)
        wide[:, :oc] = res
        dr = view(DT.from_numpy(wide))
        cabi.check(cabi.lib().fml_conv_residual(_ref(dx), _ref(dg), _ref(dw), _ref(db), _ref(dr), _ref(y), ctypes.byref(p), None))
    elif gate is not None:
        cabi.check(cabi.lib().fml_conv_scaled(_ref(dx), _ref(dg), _ref(dw), _ref(db), _ref(y), ctypes.byref(p), None))
    else:
        cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(dw), _ref(db), _ref(y), ctypes.byref(p), None))
    cabi.check_device()
    got = buf.numpy()
    assert (got[:, oc:] == 7.0).all()
    return got[:, :oc]


def check(got, x, w, bias, gate, res, act):
    n, k = x.shape[0], x.shape[1]
    xs = (x * gate if gate is not None else x).reshape(n, k, -1).astype(np.float64)
    w2 = w[:, :, 0, 0].astype(np.float64)
    ref = ACTS[act](np.einsum("oi,nip->nop", w2, xs) + bias[None, :, None])
    bound = ((k + 4) * np.einsum("oi,nip->nop", np.abs(w2), np.abs(xs)) + 4 * np.abs(bias)[None, :, None]) * 2.0 ** -24 * 1.1 + 4 * np.abs(ref) * 2.0 ** -24
    if res is not None:
        ref = ref + res.reshape(ref.shape)
        bound = bound + np.abs(ref) * 2.0 ** -24
    assert (np.abs(got.reshape(ref.shape) - ref) <= bound + 1e-30).all()


@pytest.mark.gpu
@pytest.mark.parametrize("wk,split", [(0, 0), (1, 1), (2, 1), (4, 1), (8, 1), (8, 2), (8, 8)])
@pytest.mark.parametrize("n,ic,oc,h,w", [(1, 1, 4, 2, 1), (2, 3, 16, 5, 5), (1, 33, 32, 4, 8), (3, 40, 36, 7, 7), (2, 100, 24, 6, 10), (1, 257, 68, 14, 14),
                                         (2, 672, 40, 7, 7), (1, 20, 100, 16, 17), (1, 1152, 8, 4, 4), (2, 16, 32, 24, 24)])
@pytest.mark.parametrize("kind", ["plain", "gate", "gate+residual", "residual"])
def test_against_fp64(wk, split, n, ic, oc, h, w, kind):
    rng = np.random.default_rng(ic * 10 + oc)
    x, wt, bias = rng.standard_normal((n, ic, h, w)).astype(np.float32), (rng.standard_normal((oc, ic, 1, 1)) * 0.2).astype(np.float32), rng.standard_normal(oc).astype(np.float32)
    gate = rng.random((n, ic, 1, 1)).astype(np.float32) if "gate" in kind else None
    res = rng.standard_normal((n, oc, h, w)).astype(np.float32) if "residual" in kind else None
    act = [cabi.ACT_NONE, cabi.ACT_SILU, cabi.ACT_RELU][(ic + oc) % 3]
    check(run(x, wt, bias, gate, res, act, wk, split, pad=(0, 3)[oc % 8 == 0]), x, wt, bias, gate, res, act)


@pytest.mark.gpu
def test_infinities_and_nans_stay_where_they_are():
    rng = np.random.default_rng(1)
    x, w = rng.standard_normal((1, 64, 6, 6)).astype(np.float32), rng.standard_normal((32, 64, 1, 1)).astype(np.float32)
    x[0, 5, 0, 0], x[0, 6, 2, 3] = np.inf, np.nan
    got = run(x, w, np.zeros(32, np.float32), None, None, cabi.ACT_NONE)
    assert not np.isfinite(got[0, :, 0, 0]).any() and np.isnan(got[0, :, 2, 3]).all()
    rest = np.ones((6, 6), bool)
    rest[0, 0] = rest[2, 3] = False
    assert np.isfinite(got[0][:, rest]).all()


class Host:
    def __init__(self, shape, layout=None):
        self.array = np.zeros(shape, np.float32)
        self.shape, self.strides = shape, cabi.gen_strides(shape, layout)

    def c(self):
        t = cabi.Tensor()
        t.data, t.dtype, t.rank = self.array.ctypes.data, cabi.F32, len(self.shape)
        for i, (s, st) in enumerate(zip(self.shape, self.strides)):
            t.shape[i], t.stride[i] = s, st
        return t


def prefers(n, ic, oc, h, w, layout=(3, 2, 0, 1), stride=1, precision=cabi.GEMM_AUTO):
    p = params(cabi.ACT_NONE, 0, 0)
    p.pointwise_fma, p.precision = 0, precision
    p.strides[0] = p.strides[1] = stride
    out = ctypes.c_int()
    x, wt, y = Host((n, ic, h, w)), Host((oc, ic, 1, 1), list(layout)), Host((n, oc, (h - 1) // stride + 1, (w - 1) // stride + 1))
    cabi.check(cabi.lib().fml_conv_prefers_fma(_ref(x), _ref(wt), _ref(y), ctypes.byref(p), 0, ctypes.byref(out)))
    return bool(out.value)


def test_the_rule():
    assert prefers(1, 96, 24, 56, 56) and prefers(1, 672, 192, 4, 4) and prefers(1, 32, 16, 112, 112)
    assert not prefers(64, 96, 24, 56, 56) and not prefers(16, 320, 1280, 7, 7)      # much arithmetic: tensor cores
    assert not prefers(1, 96, 24, 56, 56, layout=(0, 1, 2, 3))                       # weights as ONNX stores them
    assert not prefers(1, 96, 24, 56, 56, stride=2) and not prefers(1, 96, 24, 56, 56, precision=cabi.GEMM_3XTF32)
    assert not prefers(1, 96, 23, 56, 56)


@pytest.mark.gpu
@pytest.mark.parametrize("image", [32, 64, 128])
def test_small_images_through_the_executor(image):
    from oracle import oracle as orc
    model = models.build_efficientnet_b0(batch=2, image=image, std=0.16)
    x = models.efficientnet_inputs(batch=2, image=image)
    out = {o.name: np.zeros(o.shape, np.float32) for o in model.outputs}
    Executor.make_dp_greedy("t").compile(model.to_bytes()).invoke({**x, **out})
    for k, ref in orc.run_model(model, x, acc64=True).items():
        assert np.abs(out[k] - ref).max() <= 1e-4 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("constant", [0, 1])
def test_weights_of_an_earlier_launch(constant):
    """Weights that the launch in front writes are read when it has finished; constant ones may be on their way before."""
    rng = np.random.default_rng(5)
    oc, ic, hw = 256, 2048, 4
    x, bias = rng.standard_normal((1, ic, hw, hw)).astype(np.float32), rng.standard_normal(oc).astype(np.float32)
    weights = [rng.standard_normal((ic, oc)).astype(np.float32) for _ in range(2)]
    dx, db, dy = DT.from_numpy(x), DT.from_numpy(bias), DT((1, oc, hw, hw), np.float32)
    sources = [DT.from_numpy(np.ascontiguousarray(w.T)) for w in weights]  # (a transposing copy)
    dw = DT.from_numpy(weights[0])
    w4 = dw.view((oc, ic, 1, 1), [1, oc, 1, 1], 0)
    p = params(cabi.ACT_NONE, 0, 0)
    p.w_constant = constant
    for i in range(8):
        w = weights[i % 2 if not constant else 0]
        if not constant:
            cabi.copy_strided(sources[i % 2].view((ic, oc), [1, ic], 0), dw)
        cabi.check(cabi.lib().fml_conv(_ref(dx), _ref(w4), _ref(db), _ref(dy), ctypes.byref(p), None))
        cabi.check_device()
        check(dy.numpy(), x, w.T[:, :, None, None], bias, None, None, cabi.ACT_NONE)

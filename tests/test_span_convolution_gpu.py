"""The span-based dynamic convolution in one launch: the kernel against fp64 and the rewrite that makes it.

Tolerance: a weight is off by a few ulp (expf, a sum of at most 9 terms, a division), a sum of at most 9 products by 9
roundings more: 24 x 2^-24 of sum w|x|, which is at most the largest |x| in reach."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi, models
from fluidml_b200.cabi import DeviceTensor as DT, _ref
from fluidml_b200.executor import Executor
from fluidml_b200.onnx_lite import FLOAT


def reference(x, logits, pad):
    s, k = x.shape[1], logits.shape[3]
    w = np.exp(logits.astype(np.float64) - logits.max(-1, keepdims=True))
    w /= w.sum(-1, keepdims=True)
    xp = np.zeros((x.shape[0], s + k - 1, *x.shape[2:]))
    xp[:, pad:pad + s] = x
    return sum(w[..., j:j + 1] * xp[:, j:j + s] for j in range(k))


@pytest.mark.gpu
@pytest.mark.parametrize("taps", [3, 5, 7, 9])
@pytest.mark.parametrize("b,s,h,d", [(1, 1, 1, 4), (2, 7, 3, 32), (1, 8, 6, 64), (3, 17, 2, 6), (2, 128, 6, 64), (1, 33, 5, 1), (1, 40, 40, 8)])
@pytest.mark.parametrize("view", [False, True])
def test_against_fp64(taps, b, s, h, d, view):
    rng = np.random.default_rng(taps * 100 + s)
    x, logits = rng.standard_normal((b, s, h, d)).astype(np.float32), (rng.standard_normal((b, s, h, taps)) * 3).astype(np.float32)
    logits[0, 0, 0, 0] = -3.4028235e38
    pad = taps // 2 if s % 2 else taps - 1
    dx, dl = DT.from_numpy(x), DT.from_numpy(logits)
    if view:  # columns of a wider product, as the executor passes them; the result among others as well
        wide = np.zeros((b, s, 2 * h * d + 4), np.float32)
        wide[:, :, 4:4 + h * d] = x.reshape(b, s, -1)
        row = 2 * h * d + 4
        src = DT.from_numpy(wide)
        dx = src.view((b, s, h, d), [s * row, row, d, 1], 4)
        buf = DT.from_numpy(np.full((b, s, row), 7.0, np.float32))
        out = buf.view((b, s, h, d), [s * row, row, d, 1], h * d + 4)
    else:
        out = DT((b, s, h, d), np.float32)
    cabi.check(cabi.lib().fml_span_convolution(_ref(dx), _ref(dl), ctypes.c_int64(pad), _ref(out), None))
    cabi.check_device()
    got = out.numpy()
    if view:
        whole = buf.numpy()
        got = whole[:, :, h * d + 4:].reshape(b, s, h, d)
        assert (whole[:, :, :h * d + 4] == 7.0).all()
    assert np.abs(got - reference(x, logits, pad)).max() <= 24 * 2.0 ** -24 * np.abs(x).max()


def graph(variant="plain", taps=5, b=2, s=12, h=3, d=8):
    g = models.GraphBuilder("span")
    x, logits = g.input("x", FLOAT, (b, s, h, d)), g.input("logits", FLOAT, (b, s, h, taps))
    w = g.softmax(logits, axis=-1 if variant != "axis" else 2)
    p = g.pad(g.relu(x), [0, taps // 2, 0, 0, 0, taps // 2 + (variant == "long"), 0, 0])
    acc = None
    for j in range(taps):
        lo = j if variant != "order" or j > 1 else 1 - j
        term = g.mul(g.slice(p, [lo], [lo + s], [1]), g.slice(w, [j], [j + 1], [3]))
        acc = term if acc is None else g.add(acc, term)
    if variant == "second reader":
        acc = g.add(acc, g.slice(p, [0], [s], [1]))
    g.relu(acc, out="y")
    g.output("y")
    return g.finish()


def launches(model):
    st = Executor.make_dp_greedy("t").plan(model.to_bytes())
    return [n["kind"] for n in st["sequence"] if not n["alias"]]


def test_the_pattern_is_matched_exactly_or_not_at_all():
    ks = launches(graph())
    assert ks.count("FusedMulAddChain") == 1 and "Pad" not in ks and "Softmax" not in ks
    for variant in ("axis", "long", "order", "second reader"):
        ks = launches(graph(variant))
        assert "Pad" in ks and "Softmax" in ks
    assert "Softmax" in launches(graph(taps=4)) and "Softmax" in launches(graph(taps=11))
    conv = launches(models.build_convbert(layers=2, hidden=256, heads=8, ffn=512, vocab=400, batch=3, seq=48))
    assert conv.count("FusedMulAddChain") == 2 and "Pad" not in conv and "Softmax" not in conv


@pytest.mark.gpu
@pytest.mark.parametrize("variant", ["plain", "axis", "long", "order", "second reader"])
@pytest.mark.parametrize("make", [Executor.make_dp_greedy, Executor.make_plain_greedy])
def test_through_the_executor(variant, make):
    from oracle import oracle as orc
    model = graph(variant)
    rng = np.random.default_rng(3)
    x = {"x": rng.standard_normal((2, 12, 3, 8)).astype(np.float32), "logits": rng.standard_normal((2, 12, 3, 5)).astype(np.float32)}
    out = {"y": np.zeros((2, 12, 3, 8), np.float32)}
    make("t").compile(model.to_bytes()).invoke({**x, **out})
    assert np.abs(out["y"] - orc.run_model(model, x, acc64=True)["y"]).max() <= 24 * 2.0 ** -24 * 4

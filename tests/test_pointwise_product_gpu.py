"""A 1-D pointwise convolution between transposes as the product it is.

Tolerance: pairs hold 22 bits of each operand and drop the product of the two low parts, 3 * 2^-22 of sum|x w|; fp32
accumulation over K adds K 2^-24, the depthwise layer's three products and sums 4 * 2^-24."""
import numpy as np
import pytest

from fluidml_b200 import models
from fluidml_b200.executor import Executor


def net(b, ic, length, oc, bias=True, relu=False, read_twice=False, kernel=1, depthwise=True):
    g = models.GraphBuilder("pointwise")
    rng = np.random.default_rng(ic + length + oc)
    d = rng.standard_normal((ic, 1, 3)).astype(np.float32)
    w = rng.standard_normal((oc, ic, kernel)).astype(np.float32)
    c = rng.standard_normal(oc).astype(np.float32)
    y = g.transpose(g.input("x", 1, (b, length, ic)), [0, 2, 1])
    if depthwise:
        y = g.conv(y, g.const("d", d), None, pads=[1, 1], strides=[1], dilations=[1], group=ic)
    y = g.conv(y, g.const("w", w), g.const("c", c) if bias else None, pads=[0, 0], strides=[1], dilations=[1])
    y = g.relu(y) if relu else y
    g.output(g.neg(g.transpose(y, [0, 2, 1]), "out"))
    if read_twice:
        g.output(g.sqrt(y, "more"))
    return g.finish(), d, w, c if bias else np.zeros(oc, np.float32)


def products(*a, make=Executor.make_dp_greedy, **k):
    st = make("t").plan(net(*a, **k)[0].to_bytes())
    return sum(n["kind"] == "FusedGemm" for n in st["sequence"])


def test_which_become_products():
    assert products(2, 64, 32, 64) == 1 and products(1, 32, 64, 96, bias=False) == 1
    assert products(2, 64, 30, 64) == 0 and products(2, 64, 28, 64) == 0   # what the packed convolution does not take
    assert products(2, 64, 32, 60) == 0 and products(2, 28, 32, 64) == 0 and products(2, 64, 32, 66) == 0
    assert products(2, 64, 32, 64, relu=True) == 0 and products(2, 64, 32, 64, read_twice=True) == 0
    assert products(2, 64, 34, 64, kernel=3) == 0 and products(2, 64, 32, 64, depthwise=False) == 0
    assert products(2, 64, 32, 64, make=Executor.make_plain_greedy) == 0  # no other layouts there


@pytest.mark.gpu
@pytest.mark.parametrize("b,ic,length,oc,bias", [(1, 32, 32, 64, True), (3, 64, 36, 68, False), (2, 100, 48, 96, True), (8, 256, 128, 128, True), (1, 768, 512, 384, True)])
def test_the_numbers(b, ic, length, oc, bias):
    m, d, w, c = net(b, ic, length, oc, bias)
    x = np.random.default_rng(0).standard_normal((b, length, ic)).astype(np.float32)
    out = {"out": np.zeros((b, length, oc), np.float32)}
    Executor.make_dp_greedy("t").compile(m.to_bytes()).invoke({"x": x, **out})

    def both(f):
        wide = np.pad(f(x.astype(np.float64)), ((0, 0), (1, 1), (0, 0)))
        y = sum(wide[:, k:k + length] * f(d[:, 0, k].astype(np.float64)) for k in range(3))
        return y, y @ f(w[:, :, 0].astype(np.float64)).T

    ref, total = -(both(lambda t: t)[1] + c), both(np.abs)[1]
    off = ((3 * 2.0 ** -22 + ic * 2.0 ** -24) + 4 * 2.0 ** -24) * total + 2.0 ** -23 * np.abs(c)
    assert (np.abs(out["out"] - ref) <= off).all()

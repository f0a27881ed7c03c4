"""GPU parity of the half-precision-pair convolution (packed weights) against an fp64 convolution: every
source of the raw patch (boxes, flattened rows, plane runs, whole small planes, flattened channel and
tap), ragged tiles and channel tails, split-K, the input gate, and inputs whose first channel block
misjudges the scale of the rest (the kernel then repeats the tile)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT


def run(x, w, bias=None, pad=0, gate=None, act=cabi.ACT_NONE):
    n, _, h, wd = x.shape
    oc, _, k, _ = w.shape
    dx, dw, y = DT.from_numpy(x), DT.from_numpy(w, [3, 2, 0, 1]), DT((n, oc, h + 2 * pad - k + 1, wd + 2 * pad - k + 1), np.float32)
    assert cabi.conv_uses_packed(dx, dw, y, [pad, pad], scaled=gate is not None)
    packed = cabi.conv_pack(dw)
    db = None if bias is None else DT.from_numpy(bias)
    if gate is None:
        cabi.conv(dx, dw, db, y, [pad, pad], [1, 1], [1, 1], act=act, packed=packed)
    else:
        cabi.conv_scaled(dx, DT.from_numpy(gate), dw, db, y, [pad, pad], [1, 1], [1, 1], act=act, packed=packed)
    cabi.check_device()
    return y.numpy()


def reference(x, w, bias=None, pad=0, gate=None):
    t = lambda a: torch.from_numpy(a.astype(np.float64))
    xs = x if gate is None else (x * gate).astype(np.float32)
    return torch.nn.functional.conv2d(t(xs), t(w), None if bias is None else t(bias), padding=pad).numpy()


@pytest.mark.parametrize("n,ic,oc,h,w,k,pad", [
    (2, 32, 64, 24, 40, 3, 1), (1, 48, 36, 17, 20, 3, 1), (1, 64, 128, 16, 8, 3, 1), (1, 40, 32, 21, 12, 5, 2),  # boxes
    (2, 64, 96, 14, 14, 3, 1), (1, 96, 512, 10, 10, 3, 1), (1, 512, 512, 14, 14, 3, 1),                          # flattened rows
    (3, 16, 96, 20, 20, 1, 0), (1, 100, 24, 28, 28, 1, 0), (1, 320, 1280, 14, 14, 1, 0), (2, 24, 144, 56, 56, 1, 0),  # runs
    (7, 192, 320, 7, 7, 1, 0), (2, 64, 40, 9, 9, 1, 0), (1, 1152, 192, 7, 7, 1, 0),                              # whole planes
    (2, 3, 64, 32, 32, 3, 1), (1, 6, 32, 19, 36, 3, 1), (1, 2, 16, 33, 20, 5, 2),                                # channel x tap
])
def test_shapes(n, ic, oc, h, w, k, pad):
    rng = np.random.default_rng(n * ic + oc + h)
    x = rng.standard_normal((n, ic, h, w), np.float32)
    wt = rng.standard_normal((oc, ic, k, k), np.float32) / np.float32(np.sqrt(ic * k * k))
    b = rng.standard_normal(oc, np.float32)
    ref = reference(x, wt, b, pad)
    assert np.abs(run(x, wt, b, pad) - ref).max() <= 1e-5 * np.abs(ref).max()
    assert np.abs(run(x, wt, b, pad, act=cabi.ACT_RELU) - np.maximum(ref, 0)).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("n,ic,oc,hw", [(2, 96, 24, 28), (5, 480, 112, 7)])
def test_gate(n, ic, oc, hw):
    rng = np.random.default_rng(hw)
    x, w = rng.standard_normal((n, ic, hw, hw), np.float32), rng.standard_normal((oc, ic, 1, 1), np.float32) * 0.1
    g = rng.random((n, ic, 1, 1), np.float32)
    ref = reference(x, w, gate=g)
    assert np.abs(run(x, w, gate=g) - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("ic,hw,k", [(96, 16, 3), (128, 14, 1)])
def test_scale_is_corrected(ic, hw, k):
    rng = np.random.default_rng(ic)
    w = rng.standard_normal((32, ic, k, k), np.float32)
    base = rng.standard_normal((1, ic, hw, hw), np.float32)
    for first, rest in ((1e-4, 1e3), (0.0, 1e-9), (0.0, 1e5), (1e20, 1e-3), (0.0, 0.0)):
        x = base.copy()
        x[:, :32] *= np.float32(first)
        x[:, 32:] *= np.float32(rest)
        ref, got = reference(x, w, pad=k // 2), run(x, w, pad=k // 2)
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max() + 1e-37


@pytest.mark.parametrize("ic,oc,h,w,k", [(64, 32, 128, 256, 1), (64, 512, 64, 64, 1), (96, 64, 128, 128, 3)])
def test_every_tile_is_repeated(ic, oc, h, w, k):
    """Hundreds of CTAs whose second attempt ends right after their last block is split: both attempts'
    accumulator phases are waited for in order."""
    rng = np.random.default_rng(oc)
    x, wt = rng.standard_normal((2, ic, h, w), np.float32), rng.standard_normal((oc, ic, k, k), np.float32)
    x[:, :32] = 0.0
    x[:, 32:] *= np.float32(1e6)
    ref = reference(x, wt, pad=k // 2)
    for _ in range(4):
        assert np.abs(run(x, wt, pad=k // 2) - ref).max() <= 1e-5 * np.abs(ref).max()


SOURCES = [(3, 64, 40, 24, 40, 3, 1), (3, 96, 64, 14, 14, 3, 1), (3, 40, 32, 21, 12, 5, 2), (3, 512, 64, 14, 14, 3, 1),  # boxes, flattened rows
           (3, 96, 40, 20, 20, 1, 0), (3, 320, 64, 14, 14, 1, 0), (7, 192, 96, 7, 7, 1, 0), (5, 1152, 64, 7, 7, 1, 0),  # runs, whole planes
           (3, 3, 64, 32, 32, 3, 1), (3, 6, 32, 19, 36, 3, 1), (3, 64, 32, 16, 24, 1, 1)]                               # channel x tap; 1 x 1, padded


def check_every_pixel(got, x, w, pad, gate=None, where=True):
    """8e-6 of the sum of magnitudes that the output adds up, whatever the other pixels and images hold.  (Both
    halves of a pair are rounded, 2^-22; a sum of 16 products is truncated below its largest: where one value
    outweighs the rest that is most of the error.  Measured: at most 1e-6, with outweighing values 3.7e-6; the
    3xTF32 kernel on the same inputs 1.6e-6 and 5.6e-6.)"""
    ref, size = reference(x, w, pad=pad, gate=gate), reference(np.abs(x), np.abs(w), pad=pad, gate=gate)
    assert (np.where(where, np.abs(got - ref), 0.0) <= 8e-6 * size + 1e-37).all()


@pytest.mark.parametrize("n,ic,oc,h,w,k,pad", SOURCES)
@pytest.mark.parametrize("kind", ["images", "region", "stray", "late", "ramp"])
def test_magnitudes_do_not_mix(n, ic, oc, h, w, k, pad, kind):
    rng = np.random.default_rng(h + ic)
    x, wt = rng.standard_normal((n, ic, h, w), np.float32), rng.standard_normal((oc, ic, k, k), np.float32)
    if kind == "images":  # one request of the batch is 1e6 times the others
        x[1] *= np.float32(1e6)
    elif kind == "region":
        x[:, :, : h // 2] *= np.float32(1e-6)
        x[0, :, :, w // 2:] = 0.0
    elif kind == "stray":
        x[0, 1, 2, 3], x[1, ic - 1, h - 1, w - 1], x[2, 0, 0, 0] = 1e12, -3e20, 1e30
    elif kind == "late":  # pixels that outgrow the scale in their last channel
        x[:, ic - 1, ::3, ::2] *= np.float32(1e5)
    else:
        x *= np.geomspace(1e-15, 1e15, w).astype(np.float32)
    check_every_pixel(run(x, wt, pad=pad), x, wt, pad)


@pytest.mark.parametrize("n,ic,oc,h,w,k,pad", SOURCES)
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_infinities_stay_with_the_pixels_that_touch_them(n, ic, oc, h, w, k, pad, value):
    rng = np.random.default_rng(w + ic)
    x, wt = rng.standard_normal((n, ic, h, w), np.float32), rng.standard_normal((oc, ic, k, k), np.float32)
    x[2] *= np.float32(1e-8)
    at = [(0, ic // 2, 1, 2), (1, 0, h - 2, w - 1), (2, ic - 1, 3, 3)]
    finite, touched = x.copy(), np.zeros((n, 1, h, w), np.float32)
    for i in at:
        x[i], finite[i], touched[i[0], 0, i[2], i[3]] = value, 0.0, 1.0
    hit = reference(touched, np.ones((1, 1, k, k), np.float32), pad=pad) > 0
    got = run(x, wt, pad=pad)
    assert not np.isfinite(got[np.broadcast_to(hit, got.shape)]).any()
    check_every_pixel(got, finite, wt, pad, where=~hit)


@pytest.mark.parametrize("n,ic,oc,hw", [(3, 96, 24, 28), (5, 480, 112, 7), (3, 480, 40, 14)])
def test_gates_of_one_image_leave_the_others_alone(n, ic, oc, hw):
    rng = np.random.default_rng(hw)
    x, w = rng.standard_normal((n, ic, hw, hw), np.float32), rng.standard_normal((oc, ic, 1, 1), np.float32)
    g = rng.random((n, ic, 1, 1), np.float32)
    g[1] *= np.float32(1e7)
    g[2, :40] = 0.0
    check_every_pixel(run(x, w, gate=g), x, w, 0, gate=g)


@pytest.mark.parametrize("n,ic,oc,length", [(8, 768, 384, 128), (3, 40, 100, 36), (1, 32, 64, 1000)])
def test_one_dimensional_pointwise(n, ic, oc, length):
    rng = np.random.default_rng(length)
    x, w, b = rng.standard_normal((n, ic, length), np.float32), rng.standard_normal((oc, ic, 1), np.float32) * 0.1, rng.standard_normal(oc, np.float32)
    dx, dw, y = DT.from_numpy(x), DT.from_numpy(w), DT((n, oc, length), np.float32)
    assert cabi.conv_uses_packed(dx, dw, y, [0, 0])
    cabi.conv(dx, dw, DT.from_numpy(b), y, [0], [1], [1], packed=cabi.conv_pack(dw))
    cabi.check_device()
    ref = np.einsum("oi,nil->nol", w[..., 0].astype(np.float64), x.astype(np.float64)) + b[:, None]
    assert np.abs(y.numpy() - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("n,ic,oc,hw,k,gated,layout", [
    (2, 96, 24, 28, 1, True, None), (3, 240, 40, 14, 1, True, None), (5, 1152, 192, 7, 1, True, None), (1, 64, 64, 24, 3, False, None),
    (1, 512, 512, 14, 3, False, None), (2, 96, 24, 28, 1, True, [0, 2, 3, 1])])  # the last: a residual laid out otherwise
def test_residual(n, ic, oc, hw, k, gated, layout):
    rng = np.random.default_rng(hw + oc)
    x, w = rng.standard_normal((n, ic, hw, hw), np.float32), rng.standard_normal((oc, ic, k, k), np.float32) * np.float32(0.05)
    res, b = rng.standard_normal((n, oc, hw, hw), np.float32), rng.standard_normal(oc, np.float32)
    g = rng.random((n, ic, 1, 1), np.float32) if gated else None
    dx, dw, y = DT.from_numpy(x), DT.from_numpy(w, [3, 2, 0, 1]), DT((n, oc, hw, hw), np.float32)
    cabi.conv_residual(dx, None if g is None else DT.from_numpy(g), dw, DT.from_numpy(b), DT.from_numpy(res, layout), y, [k // 2, k // 2],
                       act=cabi.ACT_RELU, packed=cabi.conv_pack(dw))
    cabi.check_device()
    ref = np.maximum(reference(x, w, b, k // 2, g), 0) + res
    assert np.abs(y.numpy() - ref).max() <= 1e-5 * np.abs(ref).max()

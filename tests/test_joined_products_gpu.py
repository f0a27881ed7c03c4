"""Products joined into one launch: several projections side by side (rotation of the first columns, activation of the
last) and two left-hand sides, against fp64 and against the parts run one by one; and the rewrites that make them.

Tolerance, of the largest magnitude.  On the packed-weight kernel 8e-6, as in its own tests (operands of 22 bits), and for more
than 600 products what cutting the accumulator to 24 bits comes to: three times per sixteen products, 2^-24 of it on average.
2e-5 where the parts run on the 3xTF32 kernel (operands of 21 to 22 truncated bits, eight products at a time), as in its tests.
A rotation or a GELU adds two roundings.
"""
import math

import numpy as np
import pytest

from fluidml_b200 import cabi, models
from fluidml_b200.cabi import DeviceTensor as DT
from fluidml_b200.executor import Executor
from fluidml_b200.onnx_lite import FLOAT

PAIRS, TF32 = 8e-6, 2e-5
pairs = lambda k: max(PAIRS, 3 * k / 16 * 2.0 ** -24 + 2.0 ** -21)
erf = np.vectorize(math.erf)


def close(got, ref, tol=PAIRS):
    return np.abs(got.astype(np.float64) - ref).max() <= tol * np.abs(ref).max()


def params(b, packed, **kw):
    p = cabi.gemm_params(act=kw.pop("act", cabi.ACT_NONE), tile_n=kw.pop("tile", 0), split_k=kw.pop("split", 0))
    blob = cabi.gemm_pack(b) if packed else None
    if packed:
        p.b_constant, p.b_packed = 1, blob.ptr
    for k, v in kw.items():
        setattr(p, k, v)
    return p, blob


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 31, 32, 33, 128, 129, 300])
@pytest.mark.parametrize("k1,k2", [(32, 32), (64, 20), (96, 160), (1024, 256), (40, 64)])
@pytest.mark.parametrize("n,tile,split", [(16, 0, 0), (96, 32, 2), (200, 256, 1), (768, 128, 8), (130, 64, 4)])
def test_two_left_hand_sides(m, k1, k2, n, tile, split):
    rng = np.random.default_rng(m * 7 + k1 + n)
    a1, a2 = rng.standard_normal((m, k1)).astype(np.float32), rng.standard_normal((m, k2)).astype(np.float32)
    a2[:: 3] *= 1e-3          # rows whose parts differ in magnitude,
    a2[1:: 4] *= 3e4          # and rows whose second part outgrows the scale of the first
    b, bias, res = (rng.standard_normal(s).astype(np.float32) for s in ((k1 + k2, n), (n,), (m, n)))
    ref = np.concatenate([a1, a2], 1).astype(np.float64) @ b + bias + res
    db, c = DT.from_numpy(b), DT((m, n), np.float32)
    wide = DT.from_numpy(np.concatenate([np.ones((m, 4), np.float32), a2], 1))  # a view with a row stride of its own
    a2v = wide.view((m, k2), [k2 + 4, 1], 4)
    for packed in (True, False):
        p, blob = params(db, packed, tile=tile if packed else 0, split=split if packed else 0)
        p.a2 = a2v.c()
        cabi.gemm(DT.from_numpy(a1), db, c, DT.from_numpy(bias), DT.from_numpy(res), p)
        cabi.check_device()
        rows = np.abs(ref).max(1, keepdims=True)  # each row by its own magnitude
        assert (np.abs(c.numpy() - ref) <= (pairs(k1 + k2) if packed else TF32) * np.maximum(rows, 1.0)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("batch,length", [(1, 5), (1, 32), (3, 77), (2, 128)])
@pytest.mark.parametrize("heads,size,rot", [(2, 64, 16), (3, 32, 32), (2, 64, 64), (2, 48, 12), (4, 16, 8)])
@pytest.mark.parametrize("tile,split", [(0, 0), (16, 1), (48, 2), (96, 4), (256, 8)])
def test_projections_side_by_side(batch, length, heads, size, rot, tile, split):
    """[Q | K | V | GELU(F)] of the same rows: rotated, plain and activated columns."""
    rng = np.random.default_rng(batch * 1000 + length + size)
    m, k, h, ffn = batch * length, 256, heads * size, 80
    a = rng.standard_normal((m, k)).astype(np.float32)
    b, bias = (rng.standard_normal((k, 3 * h + ffn)) * 0.1).astype(np.float32), rng.standard_normal(3 * h + ffn).astype(np.float32)
    ang = rng.standard_normal((length, rot))
    cos, sin = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    y = a.astype(np.float64) @ b + bias
    qk = y[:, :2 * h].reshape(batch, length, 2 * heads, size)
    x = qk[..., :rot].copy()
    half = np.concatenate([-x[..., rot // 2:], x[..., :rot // 2]], -1)
    qk[..., :rot] = x * cos[None, :, None] + half * sin[None, :, None]
    f = y[:, 3 * h:]
    ref = np.concatenate([qk.reshape(m, 2 * h), y[:, 2 * h:3 * h], f * (erf(f / np.sqrt(2.0)) + 1) * 0.5], 1)
    db, c, dc, ds = DT.from_numpy(b), DT((m, 3 * h + ffn), np.float32), DT.from_numpy(cos), DT.from_numpy(sin)
    for packed in (True, False):
        p, blob = params(db, packed, act=cabi.ACT_GELU_ERF, tile=tile if packed else 0, split=split if packed else 0, act_from=3 * h, rot=rot, rot_head=size,
                         rot_cols=2 * h, rot_len=length, rot_cos=dc.c().data, rot_sin=ds.c().data)
        cabi.gemm(DT.from_numpy(a), db, c, DT.from_numpy(bias), None, p)
        cabi.check_device()
        assert close(c.numpy(), ref, PAIRS if packed else TF32)


@pytest.mark.gpu
@pytest.mark.parametrize("split", [3, 5, 6, 7])
def test_rotation_with_splits_that_are_no_power_of_two(split):
    """Their epilogue goes element by element and does not rotate: the rotation is a launch of its own."""
    rng = np.random.default_rng(split)
    length, heads, size, rot, k = 64, 2, 32, 16, 256
    m, n = 2 * length, 3 * heads * size
    a, b, bias = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (n,)))
    ang = rng.standard_normal((length, rot))
    cos, sin = np.cos(ang).astype(np.float32), np.sin(ang).astype(np.float32)
    ref = a.astype(np.float64) @ b + bias
    qk = ref[:, :2 * heads * size].reshape(2, length, 2 * heads, size)
    x = qk[..., :rot].copy()
    qk[..., :rot] = x * cos[None, :, None] + np.concatenate([-x[..., rot // 2:], x[..., :rot // 2]], -1) * sin[None, :, None]
    ref[:, :2 * heads * size] = qk.reshape(m, -1)
    db, c, dc, ds = DT.from_numpy(b), DT((m, n), np.float32), DT.from_numpy(cos), DT.from_numpy(sin)
    p, blob = params(db, True, tile=64, split=split, rot=rot, rot_head=size, rot_cols=2 * heads * size, rot_len=length,
                     rot_cos=dc.c().data, rot_sin=ds.c().data)
    cabi.gemm(DT.from_numpy(a), db, c, DT.from_numpy(bias), None, p)
    cabi.check_device()
    assert close(c.numpy(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("act_from", [1, 50, 63, 95])
@pytest.mark.parametrize("tile,split,residual", [(32, 1, False), (48, 1, False), (64, 2, False), (96, 1, True)])
def test_activation_from_any_column(act_from, tile, split, residual):
    """Column groups of four that the activation begins inside, in either ending of the kernel."""
    rng = np.random.default_rng(act_from + tile)
    m, n, k = 129, 96, 128
    a, b, bias, res = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (n,), (m, n)))
    ref = a.astype(np.float64) @ b + bias
    f = ref[:, act_from:]
    ref[:, act_from:] = f * (erf(f / np.sqrt(2.0)) + 1) * 0.5
    if residual:
        ref += res
    db, c = DT.from_numpy(b), DT((m, n), np.float32)
    p, blob = params(db, True, act=cabi.ACT_GELU_ERF, tile=tile, split=split, act_from=act_from)
    cabi.gemm(DT.from_numpy(a), db, c, DT.from_numpy(bias), DT.from_numpy(res) if residual else None, p)
    cabi.check_device()
    assert close(c.numpy(), ref)


def refused(a, b, c, **kw):
    p = cabi.gemm_params(act=kw.pop("act", cabi.ACT_NONE))
    for k, v in kw.items():
        setattr(p, k, v)
    with pytest.raises(cabi.FmlError):
        cabi.gemm_plan(a, b, c, p)


class Host:
    """A tensor of host memory: planning looks at shapes, strides and addresses only."""
    def __init__(self, *shape):
        self.array = np.zeros(shape, np.float32)
        self.shape = shape

    def c(self):
        t = cabi.Tensor()
        t.data, t.dtype, t.rank = self.array.ctypes.data, cabi.F32, len(self.shape)
        for i, (s, st) in enumerate(zip(self.shape, self.array.strides)):
            t.shape[i], t.stride[i] = s, st // 4
        return t


def test_what_does_not_chain_is_refused():
    a, b, c, a2, t = Host(64, 32), Host(96, 48), Host(64, 48), Host(64, 64), Host(64, 16)
    rot = dict(rot=16, rot_head=16, rot_cols=32, rot_len=64, rot_cos=t.array.ctypes.data, rot_sin=t.array.ctypes.data)
    refused(a, b, c, a2=Host(64, 60).c())                      # columns do not add up
    refused(a, b, c, a2=Host(63, 64).c())                      # other rows
    refused(a, b, c, a2=a2.c(), act=cabi.ACT_RELU)
    refused(a, b, c, a2=a2.c(), alpha=2.0)
    a = Host(64, 96)
    refused(a, b, c, act_from=48, act=cabi.ACT_GELU_ERF)       # no such column
    refused(a, b, c, act=cabi.ACT_GELU_ERF, **rot)             # an activation on rotated columns
    refused(a, b, c, **{**rot, "rot_cols": 40})                # part of a head
    refused(a, b, c, **{**rot, "rot_len": 60})                 # rows are no multiple of the tables'
    refused(a, b, c, **{**rot, "rot_cos": None})
    cabi.gemm_plan(a, b, c, cabi.gemm_params())


def block(m, gamma_seed, rows=2):
    """Two LayerNorms of x with scales and shifts of their own: (x + gelu(ln2(x) W1 + b1) W2) + ln1(x) W3."""
    rng = np.random.default_rng(gamma_seed)
    g = models.GraphBuilder("block")
    x = g.input("x", FLOAT, (rows, m, 64))
    f32 = lambda *s, scale=0.1: (rng.standard_normal(s) * scale).astype(np.float32)
    ln = lambda i: g.layernorm(x, g.const(f"g{i}", 1 + f32(64, scale=0.5)), g.const(f"b{i}", f32(64, scale=0.5)), -1, 1e-5)
    h1, h2 = ln(1), ln(2)
    f = g.add(g.const("c1", f32(96)), g.matmul(h2, g.const("w1", f32(64, 96))))
    e = g.erf(g.div(f, g.scalar(math.sqrt(2.0))))
    f = g.mul(g.mul(f, g.add(e, g.scalar(1.0))), g.scalar(0.5))
    f = g.matmul(f, g.const("w2", f32(96, 64)))
    a = g.add(g.const("c3", f32(64)), g.matmul(h1, g.const("w3", f32(64, 64))))
    g.add(g.add(a, f), x, out="y")
    g.output("y")
    return g.finish()


def test_a_parallel_block_is_three_launches():
    kinds = [n["kind"] for n in Executor.make_plain_greedy("t").plan(block(40, 0).to_bytes())["sequence"]]
    assert kinds.count("LayerNormalizationConstantScaleBias") == 1 and kinds.count("FusedGemm") == 2
    few = [n["kind"] for n in Executor.make_plain_greedy("t").plan(block(5, 0).to_bytes())["sequence"]]
    assert few.count("FusedGemm") == 3 and few.count("LayerNormalizationConstantScaleBias") == 2  # ten rows: as before
    exact = [n["kind"] for n in Executor.make_plain_greedy("t").set_option("gemm_precision", "fp32").plan(block(40, 0).to_bytes())["sequence"]]
    assert exact.count("FusedGemm") == 3


@pytest.mark.gpu
@pytest.mark.parametrize("m", [5, 16, 17, 77])
@pytest.mark.parametrize("make", [Executor.make_dp_greedy, Executor.make_plain_greedy])
def test_a_parallel_block_against_the_oracle(m, make):
    from oracle import oracle as orc
    model = block(m, m)
    x = {"x": np.random.default_rng(1).standard_normal((2, m, 64)).astype(np.float32)}
    out = {"y": np.zeros((2, m, 64), np.float32)}
    make("t").compile(model.to_bytes()).invoke({**x, **out})
    assert close(out["y"], orc.run_model(model, x, acc64=True)["y"])


@pytest.mark.gpu
@pytest.mark.parametrize("k1,k2", [(32, 64), (96, 20), (20, 64)])
@pytest.mark.parametrize("m", [3, 40, 140])
def test_a_concatenation_in_front_of_a_product(k1, k2, m):
    from oracle import oracle as orc
    rng = np.random.default_rng(k1 + m)
    g = models.GraphBuilder("cat")
    a, b = g.input("a", FLOAT, (m, k1)), g.input("b", FLOAT, (m, k2))
    w = g.const("w", rng.standard_normal((k1 + k2, 48)).astype(np.float32))
    g.matmul(g.concat(g.relu(a), g.relu(b), 1), w, out="y")
    g.output("y")
    model = g.finish()
    x = {"a": rng.standard_normal((m, k1)).astype(np.float32), "b": rng.standard_normal((m, k2)).astype(np.float32)}
    out = {"y": np.zeros((m, 48), np.float32)}
    ex = Executor.make_dp_greedy("t").compile(model.to_bytes())
    ex.invoke({**x, **out})
    assert close(out["y"], orc.run_model(model, x, acc64=True)["y"])


def two_halves(apart, top, rows=64, k1=256, k2=512, n=64):
    """(a1 W1 + a2 W2) + x whose halves contribute alike, W of one half (0: the first) `apart` times the other's."""
    rng = np.random.default_rng(int(np.log2(apart)) * 2 + top)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    w1, w2, feeds = f32(k1, n), f32(k2, n), {"a1": f32(rows, k1), "a2": f32(rows, k2), "x": f32(rows, n)}
    if top:
        w2, feeds["a2"] = w2 * np.float32(apart), feeds["a2"] / np.float32(apart)
    else:
        w1, feeds["a1"] = w1 * np.float32(apart), feeds["a1"] / np.float32(apart)
    g = models.GraphBuilder("halves")
    a1, a2, x = (g.input(name, FLOAT, v.shape) for name, v in feeds.items())
    g.add(g.add(g.matmul(a1, g.const("w1", w1)), g.matmul(a2, g.const("w2", w2))), x, out="y")
    g.output("y")
    wide = {k: v.astype(np.float64) for k, v in feeds.items()}
    ref = wide["a1"] @ w1 + wide["a2"] @ w2 + wide["x"]
    size = np.abs(wide["a1"]) @ np.abs(w1) + np.abs(wide["a2"]) @ np.abs(w2) + np.abs(wide["x"])
    return g.finish(), feeds, ref, size


def products(model):
    return [n["kind"] for n in Executor.make_plain_greedy("t").plan(model.to_bytes())["sequence"]].count("FusedGemm")


@pytest.mark.parametrize("top", [0, 1])
def test_halves_are_joined_where_their_weights_are_of_one_magnitude(top):
    assert products(two_halves(1, top)[0]) == 1
    assert products(two_halves(2, top)[0]) == 1
    for apart in (2.0 ** 6, 2.0 ** 12, 2.0 ** 20):
        assert products(two_halves(apart, top)[0]) == 2
    # one column is enough
    rng = np.random.default_rng(0)
    w = [rng.standard_normal((64, 64)).astype(np.float32) for _ in range(2)]
    w[top][:, 17] = 0.0
    g = models.GraphBuilder("column")
    a, b, x = (g.input(name, FLOAT, (64, 64)) for name in "abx")
    g.add(g.add(g.matmul(a, g.const("w1", w[0])), g.matmul(b, g.const("w2", w[1]))), x, out="y")
    g.output("y")
    assert products(g.finish()) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("top", [0, 1])
@pytest.mark.parametrize("apart", [1.0, 2.0, 2.0 ** 6, 2.0 ** 12, 2.0 ** 20])
def test_halves_that_differ_in_magnitude(apart, top):
    """Operands of 22 bits are off by 2^-22 each.  An accumulator takes sixteen products at a time, three times over, and
    each time cuts its sum to 24 bits: 2^-23 of it.  Bias and residual round twice more."""
    model, feeds, ref, size = two_halves(apart, top)
    out = {"y": np.zeros(ref.shape, np.float32)}
    Executor.make_dp_greedy("t").compile(model.to_bytes()).invoke({**feeds, **out})
    steps = 3 * (256 + 512) // 16
    assert (np.abs(out["y"] - ref) <= (2.0 ** -21 + (steps + 2) * 2.0 ** -23) * size).all()


def two_norms(grow, gains, rows=64, k=128, n=64):
    """ln1(x) W1 and ln2(x) W2 where two features of x, of opposite sign, are `grow` times the others and the norms' gains there as given."""
    rng = np.random.default_rng(3)
    f32 = lambda *s: rng.standard_normal(s).astype(np.float32)
    x = np.round(f32(rows, k) * 8)  # (whole numbers below 2^24: their sum, hence the mean, is exact)
    x[:, 5] = np.float32(grow) * (1 + np.minimum(np.abs(x[:, 5]), 8))
    x[:, 6] = -x[:, 5]
    g = models.GraphBuilder("norms")
    xin, ref, wide = g.input("x", FLOAT, x.shape), [], x.astype(np.float64)
    normed = (wide - wide.mean(1, keepdims=True)) / np.sqrt(wide.var(1, keepdims=True) + 1e-5)
    for i in (1, 2):
        scale = np.exp(f32(k) * 0.3).astype(np.float32)
        scale[5:7] = gains[i - 1]
        w, shift = f32(k, n), f32(k)
        h = g.layernorm(xin, g.const(f"g{i}", scale), g.const(f"b{i}", np.float32(1e-6) * shift), -1, 1e-5)
        g.add(g.const(f"c{i}", np.float32(1e-5) * shift[:n]), g.matmul(h, g.const(f"w{i}", w)), out=f"y{i}")
        g.output(f"y{i}")
        ref.append((normed * scale + 1e-6 * shift.astype(np.float64)) @ w + 1e-5 * shift[:n].astype(np.float64))
    return g.finish(), {"x": x}, ref


def norms(model):
    return [n["kind"] for n in Executor.make_plain_greedy("t").plan(model.to_bytes())["sequence"]].count("LayerNormalizationConstantScaleBias")


def test_norms_are_shared_where_their_gains_are_alike():
    for gains in ((1, 1), (2.0 ** -17, 2.0 ** -17), (0.25, 1), (-1, 1), (2.0 ** -10, 2.0 ** -13)):
        assert norms(two_norms(1, gains)[0]) == 1
    for gains in ((2.0 ** -17, 1), (0, 1), (1, 2.0 ** -9)):
        assert norms(two_norms(1, gains)[0]) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("gains", [(1, 1), (2.0 ** -17, 2.0 ** -17), (2.0 ** -17, 1), (2.0 ** -16, 2.0 ** -18)])
@pytest.mark.parametrize("grow", [1.0, 2.0 ** 14, 2.0 ** 20])
def test_norms_that_hold_features_down(grow, gains):
    """Each output by its own 2-norm: x - mean (the grown features cancel in it), its factor 1 / deviation and the gain round
    three times, the operands' halves twice more, 2^-22 together at most; 24 accumulator steps cut 2^-24 each on average."""
    model, feeds, ref = two_norms(grow, gains)
    out = {f"y{i}": np.zeros(r.shape, np.float32) for i, r in zip((1, 2), ref)}
    Executor.make_dp_greedy("t").compile(model.to_bytes()).invoke({**feeds, **out})
    for i, r in zip((1, 2), ref):
        assert np.linalg.norm(out[f"y{i}"] - r) <= (2.0 ** -22 + 24 * 2.0 ** -24) * np.linalg.norm(r)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [32, 77, 129, 300])
@pytest.mark.parametrize("k1,k2", [(32, 32), (64, 20), (512, 2048)])
@pytest.mark.parametrize("n,tile,split", [(16, 0, 0), (96, 32, 1), (260, 256, 1), (200, 192, 2), (768, 128, 8), (128, 64, 3)])
def test_sums_of_two_products(m, k1, k2, n, tile, split):
    """With a second accumulator (tiles up to 192) and without; small and large second parts, rows done twice.  Tolerance of
    two left-hand sides."""
    rng = np.random.default_rng(m + k1 + n)
    a1, a2 = rng.standard_normal((m, k1)).astype(np.float32), rng.standard_normal((m, k2)).astype(np.float32)
    a2[:: 3] *= 1e-3
    a2[1:: 4] *= 3e4
    b, bias, res = (rng.standard_normal(s).astype(np.float32) for s in ((k1 + k2, n), (n,), (m, n)))
    db, c = DT.from_numpy(b), DT((m, n), np.float32)
    for residual in (True, False):
        ref = np.concatenate([a1, a2], 1).astype(np.float64) @ b + bias + (res if residual else 0)
        p, blob = params(db, True, tile=tile, split=split)
        d2 = DT.from_numpy(a2)
        p.a2, p.summed = d2.c(), 1
        cabi.gemm(DT.from_numpy(a1), db, c, DT.from_numpy(bias), DT.from_numpy(res) if residual else None, p)
        cabi.check_device()
        rows = np.abs(ref).max(1, keepdims=True)
        assert (np.abs(c.numpy() - ref) <= pairs(k1 + k2) * np.maximum(rows, 1.0)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [40, 300, 1024, 2048])
def test_a_sum_is_no_less_exact_than_two_products(m):
    """Activations of one sign, whose sums are cut the most.  Each side with the tiles that tuning finds; two of them may be
    split differently from run to run, a factor of two in the error at most."""
    rng = np.random.default_rng(m)
    k1, k2, n = 512, 2048, 512
    a1, a2 = rng.standard_normal((m, k1)).astype(np.float32), np.abs(rng.standard_normal((m, k2))).astype(np.float32)
    b = (rng.standard_normal((k1 + k2, n)) * 0.02).astype(np.float32)
    ref = np.concatenate([a1, a2], 1).astype(np.float64) @ b
    d1, d2, db = DT.from_numpy(a1), DT.from_numpy(a2), DT.from_numpy(b)

    def product(a, w, residual=None, **kw):
        c = DT((m, n), np.float32)
        p, blob = params(w, True, **kw)
        cabi.gemm(a, w, c, None, residual, cabi.gemm_autotune(a, w, c, p, None, residual))
        cabi.check_device()
        return c

    error = lambda c: np.linalg.norm(c.numpy() - ref) / np.linalg.norm(ref)
    two = product(d2, DT.from_numpy(b[k1:].copy()), product(d1, DT.from_numpy(b[:k1].copy())))
    assert error(product(d1, db, a2=d2.c(), summed=1)) <= 2 * error(two)


def test_sums_are_joined_while_their_tiles_are_few():
    few, many = [two_halves(1, 0, rows=r, n=128)[0] for r in (64, 128 * 80)]
    assert products(few) == 1 and products(many) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("m,k", [(40, 1024), (200, 512), (77, 768)])
def test_projections_side_by_side_are_no_less_exact(m, k):
    """Rows of one sign, tuned tiles on both sides: as test_a_sum_is_no_less_exact_than_two_products."""
    rng = np.random.default_rng(m)
    n1, n2 = 3 * k, 4 * k
    a, b = np.abs(rng.standard_normal((m, k))).astype(np.float32), (rng.standard_normal((k, n1 + n2)) * 0.02).astype(np.float32)
    ref = a.astype(np.float64) @ b
    ref[:, n1:] = ref[:, n1:] * (erf(ref[:, n1:] / np.sqrt(2.0)) + 1) * 0.5
    da = DT.from_numpy(a)

    def product(w, **kw):
        dw, c = DT.from_numpy(np.ascontiguousarray(w)), DT((m, w.shape[1]), np.float32)
        p, blob = params(dw, True, **kw)
        cabi.gemm(da, dw, c, None, None, cabi.gemm_autotune(da, dw, c, p))
        cabi.check_device()
        return c.numpy()

    error = lambda y: np.linalg.norm(y[:, :n1] - ref[:, :n1]) / np.linalg.norm(ref[:, :n1])
    apart = product(b[:, :n1])
    assert error(product(b, act=cabi.ACT_GELU_ERF, act_from=n1)) <= 2 * error(apart)

"""The fused attention kernel for head sizes 32 and 64 (`attention_rows_kernel`) against fp64.

Tolerance: a score is off by at most (D / 2 + 3) 2^-24 sum|q||k| / divisor, about 1e-5 here, which is the weights'
relative error; the context adds at most 60 roundings of 2^-24.  Held to 2e-5 of the largest |v|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

LOWEST = float(np.finfo(np.float32).min)


def reference(q, k, v, mask, divisor):
    s = q.astype(np.float64) @ k.astype(np.float64).swapaxes(-1, -2) / divisor
    s = np.maximum(s + (0.0 if mask is None else mask.astype(np.float64)), LOWEST)  # fp32 has nothing below but -inf
    p = np.exp(s - s.max(-1, keepdims=True))
    return (p / p.sum(-1, keepdims=True)) @ v.astype(np.float64)


def views(q, k, v):
    """Q, K^T, V as the executor passes them: column slices of one [batch * length, 3 * heads * D] product."""
    b, h, s, d = q.shape
    row = 3 * h * d
    src = DT.from_numpy(np.concatenate([x.transpose(0, 2, 1, 3).reshape(b * s, h * d) for x in (q, k, v)], 1))
    return (src.view((b, h, s, d), [s * row, d, row, 1], 0), src.view((b, h, d, s), [s * row, d, 1, row], h * d),
            src.view((b, h, s, d), [s * row, d, row, 1], 2 * h * d))


@pytest.mark.parametrize("d", [32, 64])
@pytest.mark.parametrize("s", [1, 4, 15, 16, 17, 31, 33, 64, 77, 96, 97, 127, 128, 129, 160, 257])
@pytest.mark.parametrize("kind", ["none", "key", "full", "causal", "lowest"])
def test_against_fp64(d, s, kind):
    rng = np.random.default_rng(d * 1000 + s)
    b, h = (2, 3) if s < 200 else (1, 2)
    q, k, v = (rng.standard_normal((b, h, s, d)).astype(np.float32) for _ in range(3))
    causal, mask = False, None
    if kind == "key":
        mask = np.where(rng.random((b, 1, 1, s)) < 0.3, -10000.0, 0.0).astype(np.float32)
    elif kind == "full":
        mask = rng.standard_normal((b, h, s, s)).astype(np.float32)
    elif kind == "causal":
        causal, mask = True, np.where(np.tril(np.ones((1, 1, s, s))) > 0, 0.0, LOWEST).astype(np.float32)
    elif kind == "lowest":  # some rows see nothing at all: every score is the lowest number
        mask = np.where(rng.random((b, 1, s, s)) < 0.5, LOWEST, 0.0).astype(np.float32)
        mask[:, :, s // 2] = LOWEST
    out = DT((b * s, h * d), np.float32)
    cabi.attention(*views(q, k, v), DT.from_numpy(mask) if mask is not None else None, 8.0,
                   out.view((b, h, s, d), [s * h * d, d, h * d, 1], 0), causal=causal)
    cabi.check_device()
    got = out.numpy().reshape(b, s, h, d).transpose(0, 2, 1, 3)
    ref = reference(q, k, v, mask, 8.0)
    if kind == "lowest":  # a score of either sign vanishes beside the lowest number
        vanished = np.abs(q[:, :, s // 2, None] @ k.swapaxes(-1, -2)).max() < 1e30
        assert vanished and np.abs(got[:, :, s // 2] - v.mean(2)).max() <= 2e-5 * np.abs(v).max()
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(v).max()


def test_queries_and_keys_of_other_lengths_and_strides():
    """More queries than keys and the other way round, an output with other strides, and operands that only the
    general kernel takes (a row stride that is no multiple of four): the same result to rounding."""
    rng = np.random.default_rng(5)
    for sq, sk in ((40, 7), (9, 300), (16, 128)):
        q, k, v = (rng.standard_normal((2, 2, n, 64)).astype(np.float32) for n in (sq, sk, sk))
        ref = reference(q, k, v, None, 8.0)
        kt = DT.from_numpy(k).view((2, 2, 64, sk), [2 * sk * 64, sk * 64, 1, 64], 0)
        for layout in ([0, 1, 2, 3], [0, 1, 3, 2], [3, 1, 0, 2]):
            out = DT((2, 2, sq, 64), np.float32, layout)
            cabi.attention(DT.from_numpy(q), kt, DT.from_numpy(v), None, 8.0, out)
            cabi.check_device()
            assert np.abs(out.numpy() - ref).max() <= 2e-5 * np.abs(v).max()
        wide = np.zeros((2, 2, sq, 65), np.float32)
        wide[..., :64] = q
        out = DT((2, 2, sq, 64), np.float32)
        cabi.attention(DT.from_numpy(wide).view((2, 2, sq, 64), [2 * sq * 65, sq * 65, 65, 1], 0), kt, DT.from_numpy(v), None, 8.0, out)
        cabi.check_device()
        assert np.abs(out.numpy() - ref).max() <= 2e-5 * np.abs(v).max()

"""The half-precision-pair attention kernel (head size 64): ragged rows and keys, every kind of mask, a
running maximum that keeps growing, values whose scale changes between key blocks, rows without a key."""
import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

pytestmark = pytest.mark.gpu
LOWEST = np.finfo(np.float32).min


def oracle(q, k, v, mask, divisor):
    s = q.astype(np.float64) @ np.swapaxes(k, -1, -2).astype(np.float64) / divisor
    if mask is not None:
        s = np.maximum(s + mask, LOWEST)
    s = np.exp(s - s.max(-1, keepdims=True))
    return s / s.sum(-1, keepdims=True) @ v.astype(np.float64)


@pytest.mark.parametrize("b,h,sq,sk,kind,values", [
    (16, 12, 128, 128, "key", "plain"), (4, 25, 129, 191, None, "growing"), (2, 3, 1000, 1025, "key", "steps"),
    (8, 16, 100, 300, "full", "plain"), (5, 8, 321, 321, "causal", "growing"), (3, 8, 512, 512, "causal", "steps"),
    (32, 12, 77, 77, "causal", "plain"), (2, 64, 65, 513, "hidden", "steps"), (96, 4, 3, 700, None, "plain")])
def test_attention_pair(b, h, sq, sk, kind, values):
    rng = np.random.default_rng(b * 1000 + sk)
    q, k, v = (rng.standard_normal((b, h, s, 64)).astype(np.float32) for s in (sq, sk, sk))
    if values == "growing":   # every block of keys raises the maximum
        k *= np.linspace(0.1, 6.0, sk, dtype=np.float32)[:, None]
    elif values == "steps":   # V's scale moves up and down between blocks
        v *= np.exp2(7.0 * ((np.arange(sk) // 64) % 3) - 7.0).astype(np.float32)[:, None]
    mask = None
    if kind in ("key", "hidden"):
        mask = np.where(rng.random((b, 1, 1, sk)) < 0.2, -10000.0, 0.0).astype(np.float32)
        if kind == "hidden":  # the first blocks of one sequence, and all keys of another
            mask[0, ..., :130], mask[1] = LOWEST, LOWEST
    elif kind == "full":
        mask = rng.standard_normal((1, h, sq, sk)).astype(np.float32)
    elif kind == "causal":
        mask = np.where(np.tril(np.ones((sq, sk), np.bool_)), 0.0, LOWEST).astype(np.float32)[None, None]
    kd = DT.from_numpy(k)
    strides = list(kd.strides)
    strides[-1], strides[-2] = strides[-2], strides[-1]
    qd, ktd, vd = DT.from_numpy(q), kd.view((b, h, 64, sk), strides, 0), DT.from_numpy(v)
    assert cabi.attention_uses_tensor_cores(qd, ktd, vd)
    md, ref = DT.from_numpy(mask) if mask is not None else None, oracle(q, k, v, mask, 8.0)
    for causal in ([False, True] if kind == "causal" else [False]):
        out = DT((b, h, sq, 64), np.float32)
        cabi.attention(qd, ktd, vd, md, 8.0, out, causal=causal)
        cabi.check_device()
        got = out.numpy()
        assert np.linalg.norm(got - ref) <= 8e-6 * np.linalg.norm(ref)
        assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_infinities_stay_in_their_keys_and_columns(value):
    """A key with an infinity leaves the rows that do not see it alone, a value with one the other columns."""
    rng = np.random.default_rng(5)
    b, h, s = 2, 64, 256
    q, k, v = (rng.standard_normal((b, h, s, 64)).astype(np.float32) for _ in range(3))
    k[0, 1, 70, 3] = k[1, 7, 250, 60] = v[0, 5, 100, 9] = v[1, 60, 3, 40] = value
    mask = np.where(np.tril(np.ones((s, s), np.bool_)), 0.0, LOWEST).astype(np.float32)[None, None]
    kd = DT.from_numpy(k)
    st = list(kd.strides)
    out = DT((b, h, s, 64), np.float32)
    cabi.attention(DT.from_numpy(q), kd.view((b, h, 64, s), [*st[:2], st[3], st[2]], 0), DT.from_numpy(v), DT.from_numpy(mask), 8.0, out, causal=True)
    cabi.check_device()
    got, fine = out.numpy(), np.ones((b, h, s, 64), bool)
    fine[0, 1, 70:], fine[1, 7, 250:], fine[0, 5, :, 9], fine[1, 60, :, 40] = False, False, False, False
    ref = oracle(q, np.where(np.isfinite(k), k, 0), np.where(np.isfinite(v), v, 0), mask, 8.0)
    assert not np.isfinite(got[0, 1, 70:]).any() and not np.isfinite(got[0, 5, 100:, 9]).any() and not np.isfinite(got[1, 60, 3:, 40]).any()
    assert np.abs(np.where(fine, got - ref, 0)).max() <= 2e-5 * np.abs(ref).max()

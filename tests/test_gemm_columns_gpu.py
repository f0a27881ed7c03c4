"""Products of few rows with K-major weights (`gemm_skinny_columns_kernel`) against fp64: every split of the warps between
rows and k, ragged edges, bias, residual and activation, weights declared constant or not.

Tolerance: a sum of K products in fp32, in any order, is off by at most K 2^-24 sum|a b|, two roundings more for bias and
residual; the activations' slopes are at most 1.2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32])
@pytest.mark.parametrize("k", [4, 124, 128, 132, 260, 512, 1028, 4096])
@pytest.mark.parametrize("n", [2, 4, 5, 130, 1000])
def test_against_fp64(m, k, n):
    rng = np.random.default_rng(m * 10000 + k + n)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    bias, res = rng.standard_normal(n).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    db = DT.from_numpy(np.ascontiguousarray(b.T)).view((k, n), [1, k], 0)
    c = DT((m, n + 3), np.float32).view((m, n), [n + 3, 1], 1)
    act = (cabi.ACT_NONE, cabi.ACT_RELU, cabi.ACT_TANH)[(m + k + n) % 3]
    p = cabi.gemm_params(act=act)
    p.b_constant = (m + n) % 2
    cabi.gemm(DT.from_numpy(a), db, c, DT.from_numpy(bias), DT.from_numpy(res), p)
    cabi.check_device()
    wide = DT((m, n + 3), np.float32, None, c.buf).numpy()
    y = a.astype(np.float64) @ b + bias
    off = (k + 2) * 2.0 ** -24 * (np.abs(a.astype(np.float64)) @ np.abs(b) + np.abs(bias))
    ref = {cabi.ACT_NONE: y, cabi.ACT_RELU: np.maximum(y, 0), cabi.ACT_TANH: np.tanh(y)}[act] + res
    assert (np.abs(wide[:, 1:1 + n] - ref) <= off * 1.2 + 4 * 2.0 ** -24 * (1 + np.abs(ref))).all()


def test_batches():
    rng = np.random.default_rng(0)
    a, b = rng.standard_normal((3, 2, 6, 200)).astype(np.float32), rng.standard_normal((3, 2, 9, 200)).astype(np.float32)
    db = DT.from_numpy(b).view((3, 2, 200, 9), [3600, 1800, 1, 200], 0)
    c = DT((3, 2, 6, 9), np.float32)
    cabi.gemm(DT.from_numpy(a), db, c)
    cabi.check_device()
    ref = a.astype(np.float64) @ b.swapaxes(-1, -2)
    assert np.abs(c.numpy() - ref).max() <= 202 * 2.0 ** -24 * (np.abs(a).astype(np.float64) @ np.abs(b).swapaxes(-1, -2)).max()

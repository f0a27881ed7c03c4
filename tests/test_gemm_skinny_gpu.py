"""Products of at most 32 rows: every row class of the two weight layouts, ragged columns and k slices, split k,
constant weights (fetched ahead) and unaligned rows."""
import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("k,n", [(1, 1), (127, 33), (128, 96), (130, 40), (1280, 1000), (3000, 31)])
@pytest.mark.parametrize("k_major", [False, True])
def test_skinny(m, k, n, k_major):
    rng = np.random.default_rng(m * 7 + k + n)
    a, b = rng.standard_normal((m, k), np.float32), rng.standard_normal((k, n), np.float32)
    bias, res = rng.standard_normal(n, np.float32), rng.standard_normal((m, n), np.float32)
    ref = np.maximum(a.astype(np.float64) @ b + bias, 0.0) + res
    scale = np.abs(a.astype(np.float64)) @ np.abs(b) + np.abs(bias) + np.abs(res)
    db, c = DT.from_numpy(b, [1, 0] if k_major else None), DT((m, n), np.float32)
    for constant in (0, 1):
        p = cabi.gemm_params(act=cabi.ACT_RELU)
        p.b_constant = constant
        cabi.gemm(DT.from_numpy(a), db, c, bias=DT.from_numpy(bias), residual=DT.from_numpy(res), params=p)
        cabi.check_device()
        assert (np.abs(c.numpy() - ref) <= 2e-6 * scale).all()

"""LayerNorm at the row counts and lengths where its kernel changes, against 64 bits.

Tolerance, with u = 2^-24: a lane adds up to 4 NV values and five more in the warp, so with n = 4 NV + 12 the mean is off by
n u mean|x|, the variance by a factor of 1 +- (n + 4) u; three more roundings make the normalised value, two the result."""
import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

U = 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("length", [4, 128, 132, 256, 260, 384, 512, 516, 768, 772, 1024, 1028, 2048, 2052, 4096])
@pytest.mark.parametrize("rows", [1, 148, 149, 296, 299, 2368, 2369, 2960, 2961, 4736, 4739, 7105])
@pytest.mark.parametrize("residual", [False, True])
def test_edges(rows, length, residual):
    if rows * length > 8 << 20:
        pytest.skip("the same kernel as fewer rows of that length")
    rng = np.random.default_rng(rows + length)
    wide = DT.from_numpy((rng.standard_normal((rows, length + 8)) * 3 + 1).astype(np.float32))  # rows inside wider ones
    x = wide.numpy()[:, 4:4 + length]
    r = rng.standard_normal((rows, length)).astype(np.float32)
    g, b = rng.standard_normal(length).astype(np.float32), rng.standard_normal(length).astype(np.float32)
    out = DT.from_numpy(np.full((rows + 1, length), np.nan, np.float32))
    cabi.layernorm(wide.view((rows, length), [length + 8, 1], 4), DT.from_numpy(r) if residual else None, DT.from_numpy(g), DT.from_numpy(b),
                   out.view((rows, length), [length, 1], 0), 1, 1e-5)
    cabi.check_device()
    got = out.numpy()
    assert np.isnan(got[rows]).all()
    t = (x + r if residual else x).astype(np.float64)
    mean = t.mean(1, keepdims=True)
    inv = 1 / np.sqrt(((t - mean) ** 2).mean(1, keepdims=True) + np.float64(np.float32(1e-5)))
    hat = (t - mean) * inv
    n = 4 * -(-length // 128) + 12
    off = U * (np.abs(g) * (n * np.abs(t).mean(1, keepdims=True) * inv * (1 + np.abs(hat)) + (n + 8) * np.abs(hat)) + 2 * np.abs(b))
    assert (np.abs(got[:rows] - (hat * g + b)) <= off + 1e-30).all()

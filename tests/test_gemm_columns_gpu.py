"""Products of few rows with K-major weights (`gemm_skinny_columns_kernel`) against fp64: every split of the warps between
rows and k, ragged edges, bias, residual and activation, weights declared constant or not.

Tolerance: a sum of K products in fp32, in any order, is off by at most K 2^-24 sum|a b|, two roundings more for bias and
residual; the activations' slopes are at most 1.2."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT


@pytest.mark.gpu
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


@pytest.mark.gpu
def test_batches():
    rng = np.random.default_rng(0)
    a, b = rng.standard_normal((3, 2, 6, 200)).astype(np.float32), rng.standard_normal((3, 2, 9, 200)).astype(np.float32)
    db = DT.from_numpy(b).view((3, 2, 200, 9), [3600, 1800, 1, 200], 0)
    c = DT((3, 2, 6, 9), np.float32)
    cabi.gemm(DT.from_numpy(a), db, c)
    cabi.check_device()
    ref = a.astype(np.float64) @ b.swapaxes(-1, -2)
    assert np.abs(c.numpy() - ref).max() <= 202 * 2.0 ** -24 * (np.abs(a).astype(np.float64) @ np.abs(b).swapaxes(-1, -2)).max()


def k_major(m, k, n):
    """Whether whole columns are taken, and whether weights are better stored for them, by shapes alone."""
    def tensor(shape, strides):
        t = cabi.Tensor()
        t.data, t.rank, t.dtype = 1 << 20, 2, cabi.F32
        for i in range(2):
            t.shape[i], t.stride[i] = shape[i], strides[i]
        return t
    a, b, c, uses = tensor((m, k), (k, 1)), tensor((k, n), (1, k)), tensor((m, n), (n, 1)), ctypes.c_int()
    p = cabi.gemm_params()
    cabi.check(cabi.lib().fml_gemm_uses_columns(*(ctypes.byref(t) for t in (a, b, c, p)), ctypes.byref(uses)))
    prefers = cabi.lib().fml_gemm_prefers_k_major
    return uses.value, prefers(*(ctypes.c_int64(v) for v in (m, n, k)))


def test_which_products_take_whole_columns():
    for m, k, n in ((1, 4096, 1000), (3, 768, 768), (16, 128, 512), (16, 512, 128), (31, 512, 512)):
        assert k_major(m, k, n) == (1, 1)
    for m, k, n in ((1, 256, 50304), (4, 128, 4096), (1, 768, 32768), (8, 512, 50304)):  # wide and flat: two to six times slower
        assert k_major(m, k, n) == (0, 0)
    assert k_major(17, 4096, 4096)[0] == 0 and k_major(8, 8192, 8192)[0] == 1
    assert k_major(31, 4096, 128)[1] == 0 and k_major(16, 4096, 1024)[1] == 0            # too few CTAs; never measured


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n", [(1, 256, 8192), (1, 256, 2048), (8, 512, 16384), (8, 512, 8192), (17, 4096, 768), (16, 4096, 768), (32, 4096, 768)])
def test_either_side_of_the_line(m, k, n):
    test_against_fp64(m, k, n)

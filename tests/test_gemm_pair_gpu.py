"""GPU parity of the half-precision-pair GEMM (packed weights) against an fp64 product: tile edges,
remainders of K, N and M, split-K, both storage orders of B, and rows whose magnitude outgrows the
scale their first k block chose (the kernel then repeats the tile with exact row maxima)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT


def run(a, b, k_major=False, bias=None, res=None, **kw):
    db = DT.from_numpy(b, [1, 0] if k_major else None)
    packed = cabi.gemm_pack(db)
    da, c = DT.from_numpy(a), DT((a.shape[0], b.shape[1]), np.float32)
    ctas = kw.pop("ctas", 0)
    p = cabi.gemm_params(**kw)
    p.b_constant, p.b_packed, p.ctas_per_sm = 1, packed.ptr, ctas
    assert cabi.gemm_plan(da, db, c, p).uses_packed
    d = lambda t: None if t is None else DT.from_numpy(t)
    cabi.gemm(da, db, c, bias=d(bias), residual=d(res), params=p)
    cabi.check_device()
    return c.numpy()


def check(got, a, b, extra=0.0, tol=8e-6):
    ref = a.astype(np.float64) @ b.astype(np.float64) + extra
    rows = np.abs(ref).max(axis=1, keepdims=True)
    assert np.abs(got - ref).max() / np.abs(ref).max() <= tol
    assert (np.abs(got - ref) <= tol * rows + 1e-37).all()  # every row on its own scale


@pytest.mark.parametrize("m,k,n", [(32, 16, 16), (33, 100, 48), (128, 64, 256), (129, 68, 1000), (200, 96, 80),
                                   (127, 1028, 20), (513, 260, 264)])
@pytest.mark.parametrize("k_major", [False, True])
def test_shapes(m, k, n, k_major):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k), np.float32), rng.standard_normal((k, n), np.float32) * 0.02
    bias, res = rng.standard_normal(n, np.float32), rng.standard_normal((m, n), np.float32)
    check(run(a, b, k_major, bias, res), a, b, bias.astype(np.float64) + res)


@pytest.mark.parametrize("tile_n,split_k,ctas", [(16, 1, 2), (32, 8, 2), (48, 2, 1), (64, 4, 2), (96, 8, 1), (128, 1, 1),
                                                 (192, 2, 1), (256, 1, 1)])
def test_tiles(tile_n, split_k, ctas):
    rng = np.random.default_rng(tile_n)
    a, b = rng.standard_normal((257, 1100), np.float32), rng.standard_normal((1100, 272), np.float32) * 0.02
    check(run(a, b, tile_n=tile_n, split_k=split_k, ctas=ctas), a, b)


@pytest.mark.parametrize("split_k", [1, 4])
def test_rows_and_columns_of_any_magnitude(split_k):
    rng = np.random.default_rng(7)
    a, b = rng.standard_normal((130, 768), np.float32), rng.standard_normal((768, 96), np.float32)
    a[0::4] *= np.geomspace(1e-6, 1e6, 768).astype(np.float32)  # outgrows the first block's scale
    a[1::4, :100] = 0.0                                          # the scale comes from a later block
    a[2::4] *= np.float32(1e-30)
    a[3::4] *= np.float32(1e20)
    a[7] = 0.0
    b *= np.geomspace(1e-12, 1e6, 96).astype(np.float32)
    got = run(a, b, tile_n=32, split_k=split_k)
    ref = a.astype(np.float64) @ b.astype(np.float64)
    scale = np.abs(a.astype(np.float64)) @ np.abs(b.astype(np.float64))
    assert (np.abs(got - ref) <= 4e-6 * scale + 1e-37).all()  # norm-wise per element
    assert (got[7] == 0).all()


@pytest.mark.parametrize("act", [cabi.ACT_GELU_ERF, cabi.ACT_RELU, cabi.ACT_SILU])
def test_activations_match_the_unpacked_kernel(act):
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((128, 256), np.float32), rng.standard_normal((256, 128), np.float32) * 0.1
    bias = rng.standard_normal(128, np.float32)
    got = run(a, b, bias=bias, act=act)
    c = DT((128, 128), np.float32)
    cabi.gemm(DT.from_numpy(a), DT.from_numpy(b), c, bias=DT.from_numpy(bias), params=cabi.gemm_params(act=act))
    ref = c.numpy()
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("split_k", [1, 2])
def test_long_rows_with_stretches_of_zeros_and_small_values(split_k):
    """Long k ranges: scales chosen with samples of the whole row; one row that the samples miss."""
    rng = np.random.default_rng(11)
    a, b = rng.standard_normal((70, 4100), np.float32), rng.standard_normal((4100, 64), np.float32) * 0.02
    a *= np.repeat(rng.random((70, 82)) < 0.3, 50, axis=1)
    a[:, :32] *= np.float32(1e-4)
    a[5], a[6] = 0.0, 0.0
    a[5, 4093], a[6, 1] = 3e5, 1e-5
    got = run(a, b, tile_n=64, split_k=split_k)
    scale = np.abs(a.astype(np.float64)) @ np.abs(b.astype(np.float64))
    assert (np.abs(got - a.astype(np.float64) @ b.astype(np.float64)) <= 4e-6 * scale + 1e-37).all()


@pytest.mark.parametrize("tile_n,split_k,ctas", [(32, 1, 2), (32, 4, 2), (48, 1, 2), (64, 2, 2), (96, 1, 1), (128, 1, 1), (256, 1, 1)])
def test_left_operand_larger_than_l2(tile_n, split_k, ctas):
    """134 MB of A: loads miss L2 and land out of order, over every depth of A's ring that the planner takes."""
    import torch
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((16384, 2048), np.float32), rng.standard_normal((2048, 256), np.float32) * 0.02
    da, db = torch.from_numpy(a).cuda().double(), torch.from_numpy(b).cuda().double()
    got = torch.from_numpy(run(a, b, tile_n=tile_n, split_k=split_k, ctas=ctas)).cuda()
    assert ((got - da @ db).abs() <= 4e-6 * (da.abs() @ db.abs())).all()  # norm-wise per element, as above


def test_tuning_a_large_product_is_quick():
    """Candidates far behind are dropped after one launch: 0.08 s where 32 launches of each took 0.60 s."""
    import time
    rng = np.random.default_rng(6)
    a, b = DT.from_numpy(rng.standard_normal((6144, 768), np.float32)), DT.from_numpy(rng.standard_normal((768, 3072), np.float32))
    c, packed = DT((6144, 3072), np.float32), cabi.gemm_pack(b)
    p = cabi.gemm_params()
    p.b_constant, p.b_packed = 1, packed.ptr
    cabi.gemm(a, b, c, params=p)
    cabi.check_device()
    start = time.perf_counter()
    tuned = cabi.gemm_autotune(a, b, c, p)
    assert time.perf_counter() - start < 0.3
    assert tuned.tile_n >= 128

"""Tiles of the packed-weight GEMM that leave by bulk tensor stores: ragged edges in both dims, results inside wider
buffers (nothing outside may be touched), batches, every activation.  8e-6 of the largest magnitude, as in that
kernel's own tests (test_joined_products_gpu.py says where it comes from); the activations' slopes are at most 1.2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

ACTS = {cabi.ACT_NONE: lambda y: y, cabi.ACT_RELU: lambda y: np.maximum(y, 0), cabi.ACT_TANH: np.tanh, cabi.ACT_SIGMOID: lambda y: 1 / (1 + np.exp(-y)),
        cabi.ACT_SILU: lambda y: y / (1 + np.exp(-y))}


@pytest.mark.parametrize("m", [32, 33, 127, 128, 161, 300])
@pytest.mark.parametrize("n,tile", [(16, 32), (32, 32), (36, 32), (50, 64), (96, 96), (100, 96), (260, 256), (1000, 128), (48, 48)])
@pytest.mark.parametrize("pad", [0, 12])
def test_edges(m, n, tile, pad):
    rng = np.random.default_rng(m + n)
    act = list(ACTS)[(m + n) % len(ACTS)]
    a, b, bias = (rng.standard_normal(s).astype(np.float32) for s in ((m, 100), (100, n), (n,)))
    b *= 0.1
    db = DT.from_numpy(b)
    blob = cabi.gemm_pack(db)
    width = (n + 3) // 4 * 4 + pad  # rows of C on 16-byte boundaries
    buf = DT.from_numpy(np.full((m + 2, width), 7.0, np.float32))
    c = buf.view((m, n), [width, 1], width)
    p = cabi.gemm_params(act=act, tile_n=tile, split_k=1)
    p.b_constant, p.b_packed = 1, blob.ptr
    cabi.gemm(DT.from_numpy(a), db, c, DT.from_numpy(bias), None, p)
    cabi.check_device()
    got = buf.numpy()
    ref = ACTS[act](a.astype(np.float64) @ b + bias)
    assert np.abs(got[1:m + 1, :n] - ref).max() <= 8e-6 * max(1.0, np.abs(ref).max())
    got[1:m + 1, :n] = 7.0
    assert (got == 7.0).all()


@pytest.mark.parametrize("batch", [1, 3])
def test_batches_that_do_not_fold(batch):
    rng = np.random.default_rng(batch)
    a, b = rng.standard_normal((batch, 40, 64)).astype(np.float32), rng.standard_normal((64, 96)).astype(np.float32)
    db = DT.from_numpy(b)
    blob = cabi.gemm_pack(db)
    buf = DT.from_numpy(np.full((batch, 50, 96), 7.0, np.float32))  # ten rows between the batches
    c = buf.view((batch, 40, 96), [50 * 96, 96, 1], 5 * 96)
    p = cabi.gemm_params(tile_n=32, split_k=1)
    p.b_constant, p.b_packed = 1, blob.ptr
    cabi.gemm(DT.from_numpy(a), db, c, None, None, p)
    cabi.check_device()
    got, ref = buf.numpy(), a.astype(np.float64) @ b
    assert np.abs(got[:, 5:45] - ref).max() <= 8e-6 * np.abs(ref).max()
    got[:, 5:45] = 7.0
    assert (got == 7.0).all()


def test_rows_that_are_done_twice():
    """A row that outgrows the scale of its first block repeats the tile; the stored one is the second."""
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((200, 256)).astype(np.float32), rng.standard_normal((256, 128)).astype(np.float32)
    a[::5, 40:] *= 1e6
    db = DT.from_numpy(b)
    blob = cabi.gemm_pack(db)
    c = DT((200, 128), np.float32)
    p = cabi.gemm_params(tile_n=64, split_k=1)
    p.b_constant, p.b_packed = 1, blob.ptr
    cabi.gemm(DT.from_numpy(a), db, c, None, None, p)
    cabi.check_device()
    ref = a.astype(np.float64) @ b
    assert (np.abs(c.numpy() - ref) <= 8e-6 * np.abs(ref).max(1, keepdims=True)).all()


@pytest.mark.parametrize("m,k,tile", [(128, 1024, 256), (300, 64, 32), (2500, 320, 96)])
def test_whole_tiles_done_twice(m, k, tile):
    """Every row outgrows its first block's scale: what is stored waits for the second attempt's products, one k block or many."""
    rng = np.random.default_rng(m)
    a, b, bias = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, 512), (512,)))
    a[:, 33:] *= 2e5
    db = DT.from_numpy(b)
    blob = cabi.gemm_pack(db)
    c = DT((m, 512), np.float32)
    p = cabi.gemm_params(act=cabi.ACT_RELU, tile_n=tile, split_k=1)
    p.b_constant, p.b_packed = 1, blob.ptr
    cabi.gemm(DT.from_numpy(a), db, c, DT.from_numpy(bias), None, p)
    cabi.check_device()
    ref = np.maximum(a.astype(np.float64) @ b + bias, 0)
    tol = max(8e-6, 3 * k / 16 * 2.0 ** -24 + 2.0 ** -21)  # (longer k: as test_joined_products_gpu.py)
    assert (np.abs(c.numpy() - ref) <= tol * np.abs(ref).max(1, keepdims=True)).all()

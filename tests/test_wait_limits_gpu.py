"""The failure path of the bounded waits, exercised without faulting or hanging anything: a test
hook shortens the iteration limit of every mbarrier wait in the tensor-core kernels and makes their
producers issue no loads, so that each wait of a launch runs out.  The kernel must then report the
timeout through the status word (`fml_check_device` -> FML_DEVICE_TIMEOUT), return, and leave the
context usable: the same call with the hook off gives the right result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

RNG = np.random.Generator(np.random.PCG64(99))
DEVICE_TIMEOUT = 5


def rnd(*shape):
    return RNG.standard_normal(shape).astype(np.float32)


def expect_timeout_then_recover(launch, verify, drop=1):
    lib = cabi.lib()
    cabi.check_device()  # start from a clean status word
    try:
        cabi.check(lib.fml_debug_wait_test(2000, drop))
        launch()
        with pytest.raises(cabi.FmlError) as e:
            cabi.check_device()
        assert e.value.status == DEVICE_TIMEOUT
    finally:
        cabi.check(lib.fml_debug_wait_test(0, 0))
    cabi.check_device()  # the status word was cleared by the read
    launch()
    cabi.check_device()
    verify()


def test_gemm_waits_run_out_and_the_context_survives():
    a, b = rnd(128, 768), rnd(768, 768) * 0.05
    da, db, dc = DT.from_numpy(a), DT.from_numpy(b), DT((128, 768), np.float32)
    p = cabi.gemm_params(tile_n=64, split_k=8)  # the clustered split-K path: every rank times out and still meets the barriers
    assert cabi.gemm_uses_tensor_cores(da, db, dc, p)
    ref = a.astype(np.float64) @ b.astype(np.float64)
    expect_timeout_then_recover(lambda: cabi.gemm(da, db, dc, params=p),
                                lambda: np.testing.assert_allclose(dc.numpy(), ref, atol=1e-4 * np.abs(ref).max()))


def test_conv_waits_run_out_and_the_context_survives():
    x, w, b = rnd(1, 64, 14, 14), rnd(128, 64, 3, 3) * 0.05, rnd(128)
    dx, dw, db, dy = DT.from_numpy(x), DT.from_numpy(w, [3, 2, 0, 1]), DT.from_numpy(b), DT((1, 128, 14, 14), np.float32)
    assert cabi.conv_uses_tensor_cores(dx, dw, dy, (1, 1))
    from oracle import oracle as orc
    ref = orc.conv(x, w, b, np.empty((1, 128, 14, 14), np.float32), (1, 1), (1, 1), (1, 1), 1, acc64=True)
    expect_timeout_then_recover(lambda: cabi.conv(dx, dw, db, dy, (1, 1), (1, 1), (1, 1), 1),
                                lambda: np.testing.assert_allclose(dy.numpy(), ref, atol=1e-4 * np.abs(ref).max()))


def test_attention_waits_run_out_and_the_context_survives():
    B, H, S, D = 8, 12, 128, 64
    q, k, v = rnd(B, H, S, D), rnd(B, H, S, D), rnd(B, H, S, D)
    dq, dk, dv, out = DT.from_numpy(q), DT.from_numpy(k), DT.from_numpy(v), DT((B, H, S, D), np.float32)
    st = list(dk.strides)
    st[-1], st[-2] = st[-2], st[-1]
    kt = dk.view((B, H, D, S), st, 0)
    assert cabi.attention_uses_tensor_cores(dq, kt, dv)
    s = np.einsum("bhqd,bhkd->bhqk", q.astype(np.float64), k.astype(np.float64)) / 8.0
    p = np.exp(s - s.max(-1, keepdims=True))
    ref = np.einsum("bhqk,bhkd->bhqd", p / p.sum(-1, keepdims=True), v.astype(np.float64))
    expect_timeout_then_recover(lambda: cabi.attention(dq, kt, dv, None, 8.0, out),
                                lambda: np.testing.assert_allclose(out.numpy(), ref, atol=2e-5 * np.abs(ref).max()))


def test_depthwise_waits_run_out_and_the_context_survives():
    """The pipelined depthwise kernel (one tensor-map copy per tile, two buffers): with the copies
    dropped both buffers' waits run out, every CTA leaves through the uniform outcome, and the next
    launch is correct."""
    x, w, b = rnd(2, 24, 28, 28), rnd(24, 1, 3, 3), rnd(24)
    dx, dw, db, dy = DT.from_numpy(x), DT.from_numpy(w), DT.from_numpy(b), DT((2, 24, 28, 28), np.float32)
    from oracle import oracle as orc
    ref = orc.conv(x, w, b, np.empty((2, 24, 28, 28), np.float32), (1, 1, 1, 1), (1, 1), (1, 1), 24)
    expect_timeout_then_recover(lambda: cabi.conv(dx, dw, db, dy, (1, 1), (1, 1), (1, 1), 24),
                                lambda: np.testing.assert_allclose(dy.numpy(), ref, atol=1e-5 * np.abs(ref).max()))


@pytest.mark.parametrize("drop", [1, 2])  # all loads; those of a repeated attempt, with the first one's MMAs behind it
@pytest.mark.parametrize("split_k", [1, 8])
def test_packed_gemm_waits_run_out_and_the_context_survives(split_k, drop):
    a, b = rnd(300, 1024), rnd(1024, 768) * np.float32(0.05)
    a[:, 40:] *= np.float32(1e6)  # every row outgrows the scale of its first block: in the first rank, at least
    da, db, dc = DT.from_numpy(a), DT.from_numpy(b), DT((300, 768), np.float32)
    packed = cabi.gemm_pack(db)
    p = cabi.gemm_params(tile_n=64, split_k=split_k)
    p.b_constant, p.b_packed = 1, packed.ptr
    assert cabi.gemm_plan(da, db, dc, p).uses_packed
    ref = a.astype(np.float64) @ b.astype(np.float64)
    expect_timeout_then_recover(lambda: cabi.gemm(da, db, dc, params=p),
                                lambda: np.testing.assert_allclose(dc.numpy(), ref, atol=1e-5 * np.abs(ref).max()), drop)


@pytest.mark.parametrize("n,ic,oc,hw,k,drop", [
    (*layer, drop) for layer in [(2, 64, 64, 28, 3), (1, 512, 512, 14, 3), (2, 96, 24, 28, 1), (5, 192, 64, 7, 1)] for drop in (1, 2)
] + [(1, 3, 32, 32, 3, 1)])  # (the last has one k block, whose scale is exact: nothing is repeated)
def test_packed_conv_waits_run_out_and_the_context_survives(n, ic, oc, hw, k, drop):
    import torch
    x, w = rnd(n, ic, hw, hw), rnd(oc, ic, k, k) * np.float32(0.05)
    x[:, 1] *= np.float32(1e-7)
    x[:, 8 if ic == 512 else 40:] *= np.float32(1e6)  # (512 channels: split over ranks of few blocks)
    x[:, :, : hw // 2] *= np.float32(1e-9)            # two bands where there are taps
    dx, dw, dy = DT.from_numpy(x), DT.from_numpy(w, [3, 2, 0, 1]), DT((n, oc, hw, hw), np.float32)
    packed, pad = cabi.conv_pack(dw), [k // 2, k // 2]
    ref = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(w).double(), padding=k // 2).numpy()
    expect_timeout_then_recover(lambda: cabi.conv(dx, dw, None, dy, pad, [1, 1], [1, 1], packed=packed),
                                lambda: np.testing.assert_allclose(dy.numpy(), ref, atol=1e-5 * np.abs(ref).max()), drop)


def test_dropping_repeats_leaves_the_other_kernels_alone():
    """The hook's value 2 is for the packed-weight kernels: attention, depthwise and unpacked products load as ever."""
    q, x, a, b = rnd(8, 12, 128, 64), rnd(2, 24, 28, 28), rnd(128, 256), rnd(256, 96)
    w = rnd(24, 1, 3, 3)
    dq, da, db, out, c, y = DT.from_numpy(q), DT.from_numpy(a), DT.from_numpy(b), DT(q.shape, np.float32), DT((128, 96), np.float32), DT(x.shape, np.float32)
    st = list(dq.strides)
    kt = dq.view((8, 12, 64, 128), [st[0], st[1], st[3], st[2]], 0)
    cabi.check_device()
    try:
        cabi.check(cabi.lib().fml_debug_wait_test(0, 2))
        cabi.attention(dq, kt, dq, None, 8.0, out)
        cabi.conv(DT.from_numpy(x), DT.from_numpy(w), None, y, (1, 1, 1, 1), (1, 1), (1, 1), 24)
        cabi.gemm(da, db, c)
        cabi.check_device()
    finally:
        cabi.check(cabi.lib().fml_debug_wait_test(0, 0))
    np.testing.assert_allclose(c.numpy(), a.astype(np.float64) @ b, atol=1e-4)

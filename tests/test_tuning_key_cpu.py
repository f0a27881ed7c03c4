"""What a remembered choice of tiles belongs to: the device it was timed on, and everything that decides which
launch is timed.  Pure host computation."""
import ctypes

import numpy as np
import pytest

from fluidml_b200 import cabi


def tensor(shape, strides=None, address=1 << 20):
    t = cabi.Tensor()
    t.data, t.rank, t.dtype = address, len(shape), cabi.F32
    st = strides or [int(np.prod(shape[i + 1:])) for i in range(len(shape))]
    for i, (n, s) in enumerate(zip(shape, st)):
        t.shape[i], t.stride[i] = n, s
    return t


def conv_key(device=0, residual=0, scaled=0, hw=28, act=0, ic=96, y_strides=None):
    x, w = tensor((2, ic, hw, hw)), tensor((24, ic, 1, 1), [1, 24, 24 * ic, 24 * ic])
    p = cabi.ConvParams()
    for i in range(2):
        p.strides[i] = p.dilations[i] = 1
    p.group, p.act = 1, act
    buf = ctypes.create_string_buffer(512)
    cabi.check(cabi.lib().fml_conv_tuning_key(ctypes.byref(x), ctypes.byref(w), ctypes.byref(tensor((2, 24, hw, hw), y_strides)),
                                              ctypes.byref(p), scaled, residual, device, buf, ctypes.c_size_t(512)))
    return buf.value


def gemm_key(device=0, residual=False, bias=False, m=128, act=0):
    t = tensor((m, 256)), tensor((256, 512)), tensor((m, 512))
    p = cabi.gemm_params(act=act)
    p.b_constant, p.b_packed = 1, 1 << 21
    buf = ctypes.create_string_buffer(512)
    extra = [ctypes.byref(tensor((512,))) if bias else None, ctypes.byref(tensor((m, 512))) if residual else None]
    cabi.check(cabi.lib().fml_gemm_tuning_key(*(ctypes.byref(x) for x in t), *extra, ctypes.byref(p), device, buf, ctypes.c_size_t(512)))
    return buf.value


@pytest.mark.parametrize("key,changes", [
    (conv_key, [{"device": 1}, {"residual": 1}, {"scaled": 1}, {"hw": 56}, {"act": 2}, {"ic": 64}, {"y_strides": [28 * 28 * 24, 1, 28 * 24, 24]}]),
    (gemm_key, [{"device": 3}, {"residual": True}, {"bias": True}, {"m": 256}, {"act": 1}])])
def test_every_part_of_the_signature_counts(key, changes):
    keys = [key()] + [key(**c) for c in changes]
    assert keys[0] and len(set(keys)) == len(keys) and key() == keys[0]


def test_who_may_not_choose_the_fma_kernel_has_a_key_of_its_own():
    """The same planes as a 1-D layer (packed kernel only) and as a 2-D one."""
    def key(x, w, y):
        p = cabi.ConvParams()
        for i in range(2):
            p.strides[i] = p.dilations[i] = 1
        p.group = 1
        buf = ctypes.create_string_buffer(512)
        cabi.check(cabi.lib().fml_conv_tuning_key(ctypes.byref(x), ctypes.byref(w), ctypes.byref(y), ctypes.byref(p), 0, 0, 0, buf, ctypes.c_size_t(512)))
        return buf.value
    line = key(tensor((2, 96, 64)), tensor((64, 96, 1)), tensor((2, 64, 64)))
    plane = key(tensor((2, 96, 1, 64)), tensor((64, 96, 1, 1), [1, 64, 96 * 64, 96 * 64]), tensor((2, 64, 1, 64)))
    assert line and plane and line != plane


def test_nothing_to_choose():
    assert conv_key(hw=1) == b""
    assert gemm_key(m=4) == b""

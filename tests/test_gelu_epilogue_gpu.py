"""GELU as the tensor-core GEMM kernels' epilogues compute it (`erf_fast` in csrc/kernels/gemm_epilogue.cuh), over its
whole range and against fp64.

The product under it is exact: one term per output, eleven bits times eleven bits.  What is left is the formula, 6e-7
absolute in erf in fp32 arithmetic (test_erf_formula_cpu.py), and the approximations it uses (PTX: ex2.approx 2^-22
relative, rcp.approx one ulp), together below 1e-6, so 5e-7 |v|; and 2^-23 |v| for the rounding of v / c0 and of the result.
"""
import math

import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

C0 = 1.4142135381698608
erf = np.vectorize(math.erf)


@pytest.mark.gpu
@pytest.mark.parametrize("packed,tile,split", [(True, 64, 1), (True, 64, 2), (False, 64, 1), (False, 64, 2)])
def test_gelu_over_its_range(packed, tile, split):
    m, n, k = 1024, 64, 64
    a, b = np.zeros((m, k), np.float32), np.zeros((k, n), np.float32)
    a[:, 0] = (np.arange(m) - m // 2) / 2.0 ** 6                    # -8 .. 8
    b[0] = np.concatenate([np.arange(1, n - 7) / 32.0, 2.0 ** -np.arange(2, 10)])  # 1/32 .. 56/32, and into the smallest
    v = a[:, :1].astype(np.float64) * b[:1]
    db, c = DT.from_numpy(b), DT((m, n), np.float32)
    p = cabi.gemm_params(act=cabi.ACT_GELU_ERF, tile_n=tile, split_k=split)
    if packed:
        blob = cabi.gemm_pack(db)
        p.b_constant, p.b_packed = 1, blob.ptr
    assert cabi.gemm_uses_tensor_cores(DT.from_numpy(a), db, c, p)
    cabi.gemm(DT.from_numpy(a), db, c, None, None, p)
    cabi.check_device()
    exact = v * (erf(v / C0) + 1.0) * 0.5
    assert (np.abs(c.numpy() - exact) <= (5e-7 + 2.0 ** -23) * np.abs(v)).all()

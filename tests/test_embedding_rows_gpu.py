"""Embedding with addends by whole rows against numpy, bit for bit (two sums, each rounded): widths, one and two leading
dims, any combination of addends, what only the general kernel takes, and indices out of range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT


@pytest.mark.parametrize("width", [4, 20, 128, 516, 768, 6])
@pytest.mark.parametrize("lead", [(1,), (7,), (1, 5), (3, 40)])
@pytest.mark.parametrize("addends", ["", "s", "w", "sw", "bsw", "b1", "ww"])
@pytest.mark.parametrize("layout", [None, "permuted"])
def test_against_numpy(width, lead, addends, layout):
    rng = np.random.default_rng(width + len(lead))
    table, ids = rng.standard_normal((50, width)).astype(np.float32), rng.integers(0, 50, lead).astype(np.int64)
    shapes = {"": [], "s": [(lead[-1], width)], "w": [(width,)], "sw": [(1, lead[-1], width), (width,)], "bsw": [(*lead, width), (1, width)],
              "b1": [(*lead, 1)], "ww": [(width,), (1, 1, width)]}[addends]
    shapes = [s[-(len(lead) + 1):] for s in shapes]
    adds = [rng.standard_normal(s).astype(np.float32) for s in shapes]
    ref = table[ids]
    for a in adds:
        ref = (ref + a).astype(np.float32)
    out = DT(ref.shape, np.float32, None if layout is None else list(range(1, ref.ndim)) + [0])
    d = [DT.from_numpy(a) for a in adds] + [None, None]
    cabi.embedding(DT.from_numpy(table), DT.from_numpy(ids), d[0], d[1], out)
    cabi.check_device()
    assert np.array_equal(out.numpy(), ref)


def test_indices_out_of_range_are_clamped_and_reported():
    table = np.arange(80, dtype=np.float32).reshape(10, 8)
    out = DT((3, 8), np.float32)
    cabi.embedding(DT.from_numpy(table), DT.from_numpy(np.array([-1, 4, 10], np.int64)), DT.from_numpy(np.ones(8, np.float32)), None, out)
    with pytest.raises(cabi.FmlError):
        cabi.check_device()
    assert np.array_equal(out.numpy(), table[[0, 4, 9]] + 1)

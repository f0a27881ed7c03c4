"""Pad over every storage order of input and output, with and without a padded innermost dim."""
import itertools

import numpy as np
import pytest

from fluidml_b200 import cabi
from fluidml_b200.cabi import DeviceTensor as DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,before,after", [((2, 3, 8), (0, 2, 0), (0, 1, 0)), ((2, 12, 4), (0, 0, 3), (1, 0, 0)),
                                                ((1, 7, 5), (4, 0, 1), (0, 4, 2)), ((3, 128, 64), (0, 4, 0), (0, 4, 0))])
def test_pad_layouts(shape, before, after):
    x = np.random.default_rng(0).standard_normal(shape, np.float32)
    ref = np.pad(x, list(zip(before, after)))
    for li, lo in itertools.product(itertools.permutations(range(3)), repeat=2):
        out = DT(ref.shape, np.float32, list(lo))
        cabi.pad(DT.from_numpy(x, list(li)), out, before)
        cabi.check_device()
        assert (out.numpy() == ref).all(), (li, lo)

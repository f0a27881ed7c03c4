"""Both residuals of a parallel block ride in its two products: the rewrite, and its result against the oracle."""
import numpy as np
import pytest

from fluidml_b200 import models
from fluidml_b200.executor import Executor
from fluidml_b200.onnx_lite import FLOAT


def parallel_block(m, second_reader):
    """y = (x W1 W2 + x W3) + x; with `second_reader` the inner sum is an output too, and its Add has to stay."""
    rng = np.random.default_rng(m)
    g = models.GraphBuilder("parallel")
    x = g.input("x", FLOAT, (2, m, 64))
    w = [g.const(f"w{i}", (rng.standard_normal(s) * 0.1).astype(np.float32)) for i, s in enumerate([(64, 96), (96, 64), (64, 64)])]
    f = g.matmul(g.matmul(x, w[0]), w[1])
    s = g.add(f, g.matmul(x, w[2]), out="s" if second_reader else None)
    g.add(s, x, out="y")
    g.output("y")
    if second_reader:
        g.output("s")
    return g.finish()


@pytest.mark.parametrize("second_reader,adds", [(False, 0), (True, 1)])
def test_rewrite(second_reader, adds):
    ex = Executor.make_plain_greedy("t")
    kinds = [n["kind"] for n in ex.plan(parallel_block(40, second_reader).to_bytes())["sequence"]]
    assert kinds.count("AddCommon") == adds


@pytest.mark.gpu
@pytest.mark.parametrize("m", [5, 40, 300])
@pytest.mark.parametrize("second_reader", [False, True])
def test_result(m, second_reader):
    from oracle import oracle as orc
    model = parallel_block(m, second_reader)
    x = {"x": np.random.default_rng(1).standard_normal((2, m, 64)).astype(np.float32)}
    ex = Executor.make_dp_greedy("t")
    ex.compile(model.to_bytes())
    outs = {o.name: np.zeros(o.shape, np.float32) for o in model.outputs}
    ex.invoke({**x, **outs})
    for k, ref in orc.run_model(model, x).items():
        assert np.abs(outs[k] - ref).max() <= 2e-5 * np.abs(ref).max()

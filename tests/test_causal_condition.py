"""A Where between the scores and their softmax makes an attention block causal only when its condition is
lower-triangular over the scores' own last two dims: smaller conditions broadcast and hide whole rows, whole
columns or nothing."""
import numpy as np
import pytest

from fluidml_b200 import models
from fluidml_b200.executor import Executor
from fluidml_b200.onnx_lite import FLOAT

S = 128
TRIL = np.tril(np.ones((S, S), bool))
CONDITIONS = {"tril": (TRIL[None, None], True), "tril_rank_2": (TRIL, True), "one_true": (np.ones((1, 1, 1, 1), bool), False),
              "one_true_rank_2": (np.ones((1, 1), bool), False), "rows": ((np.arange(S) % 5 != 3).reshape(1, 1, S, 1), False),
              "keys": ((np.arange(S) <= 90).reshape(1, 1, 1, S), False), "diagonal_hidden": (np.tril(TRIL, -1)[None, None], False),
              "one_key_more": ((TRIL | np.eye(S, k=1, dtype=bool))[None, None], False)}


def block(cond, batch=8, heads=16):
    g = models.GraphBuilder("where")
    q, k, v = (g.input(n, FLOAT, (batch, heads, S, 64)) for n in "qkv")
    s = g.div(g.matmul(q, g.transpose(k, [0, 1, 3, 2])), g.scalar(8.0))
    s = g.where(g.const("cond", cond), s, g.scalar(models.F32_LOWEST))
    g.matmul(g.softmax(s), v, out="y")
    g.output("y")
    return g.finish()


@pytest.mark.parametrize("name", CONDITIONS)
def test_plan(name):
    cond, causal = CONDITIONS[name]
    nodes = Executor.make_plain_greedy("t").plan(block(cond).to_bytes())["sequence"]
    assert [n.get("causal", False) for n in nodes if n["kind"] == "FusedAttention"] == [causal]


@pytest.mark.gpu
@pytest.mark.parametrize("name", CONDITIONS)
def test_result(name):
    from oracle import oracle as orc
    rng = np.random.default_rng(len(name))
    model = block(CONDITIONS[name][0])  # 537 Mflop: the tensor cores' size
    x = {n: rng.standard_normal((8, 16, S, 64)).astype(np.float32) for n in "qkv"}
    y = np.zeros((8, 16, S, 64), np.float32)
    Executor.make_dp_greedy("t").compile(model.to_bytes()).invoke({**x, "y": y})
    ref = orc.run_model(model, x)["y"]
    assert np.abs(y - ref).max() <= 2e-5 * np.abs(ref).max()

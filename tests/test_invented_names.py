"""Tensors of the compiler's own making (merged weights, rows of rotary tables, plane sums, additive masks) and the scratch
of nodes beside tensors of the model that have the same names: the plan is the one without them, and so are the results."""
import numpy as np
import pytest

from fluidml_b200 import models
from fluidml_b200.executor import Executor

CASES = {
    "gpt_neox": lambda: (models.build_gpt_neox(layers=2, hidden=128, heads=2, ffn=256, vocab=100, batch=2, seq=20), models.gpt_neox_inputs(batch=2, seq=20, vocab=100)),
    "convbert": lambda: (models.build_convbert(layers=2, hidden=128, heads=4, ffn=256, vocab=100, batch=2, seq=32), models.convbert_inputs(batch=2, seq=32, vocab=100)),
    "efficientnet": lambda: (models.build_efficientnet_b0(batch=1, image=64, std=0.16),
                             {"input": np.random.default_rng(0).standard_normal((1, 3, 64, 64)).astype(np.float32)}),
}


def region_table(model, tmp_path):
    """Stats of the plan and (name, rest of the line) of every tensor in it."""
    path = tmp_path / "regions.txt"
    stats = Executor.make_dp_greedy("t").plan(model.to_bytes(), llvm=str(path))
    return stats, [line.split(" ", 1) for line in path.read_text().splitlines()]


def own_names(model):
    return {v.name for v in (*model.inputs, *model.outputs, *model.value_info)} | set(model.initializers)


def rename(model, to):
    name = lambda n: to.get(n, n)
    for v in (*model.inputs, *model.outputs, *model.value_info):
        v.name = name(v.name)
    model.initializers = {name(k): v for k, v in model.initializers.items()}
    for n in model.nodes:
        n.inputs, n.outputs = [name(i) for i in n.inputs], [name(o) for o in n.outputs]
    return model


def collided(make, tmp_path):
    """The model with as many of its tensors as possible called what the compiler would call its own."""
    model, feeds = make()
    stats, table = region_table(model, tmp_path)
    mine = own_names(model)
    invented = [(n, rest) for n, rest in table if n not in mine] + [(n["name"], " arena+") for n in stats["sequence"] if n["scratch"] and n["name"] not in mine]
    assert invented
    to, outputs = {}, [o.name for o in model.outputs]
    victims = {kind: [n for n, rest in table if n in mine and kind in rest and n not in outputs and n not in feeds] for kind in ("arena+", "constant")}
    for name, rest in invented:
        kind = "constant" if rest.endswith(" constant") else "arena+"
        if victims[kind]:
            to[victims[kind].pop()] = name
    return stats, table, rename(model, to), feeds, to


@pytest.mark.parametrize("which", CASES)
def test_the_plan_is_the_same(which, tmp_path):
    stats, table, model, _, to = collided(CASES[which], tmp_path)
    st, tb = region_table(model, tmp_path)
    names = [n for n, _ in tb]
    assert len(set(names)) == len(names) == len(table) and set(to.values()) <= set(names)
    assert [n["kind"] for n in st["sequence"]] == [n["kind"] for n in stats["sequence"]]
    assert st["peak_arena_bytes"] == stats["peak_arena_bytes"]


def test_an_output_may_have_any_name(tmp_path):
    model, _ = CASES["gpt_neox"]()
    merged = [n for n, _ in region_table(model, tmp_path)[1] if n.endswith("_merged")]
    st, tb = region_table(rename(model, {model.outputs[0].name: merged[0]}), tmp_path)
    lines = dict(tb)
    assert len(lines) == len(tb) and lines[merged[0]].endswith(" output") and st["sequence"][-1]["output"] == merged[0]


@pytest.mark.gpu
@pytest.mark.parametrize("which", CASES)
def test_the_results_are_the_same(which, tmp_path):
    _, _, model, feeds, _ = collided(CASES[which], tmp_path)
    got = []
    for m in (CASES[which]()[0], model):
        out = {o.name: np.zeros(o.shape, np.float32) for o in m.outputs}
        Executor.make_dp_greedy("t").set_option("autotune", "0").compile(m.to_bytes()).invoke({**feeds, **out})
        got.append(out)
    for name, v in got[0].items():
        assert np.array_equal(got[1][name], v)

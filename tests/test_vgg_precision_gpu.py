"""The whole VGG-16 against fp64.  Its inputs to every contraction are ReLU outputs, all of one sign, so what
a kernel truncates adds up instead of averaging out: this is the network that shows a less precise kernel first."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from fluidml_b200 import models
from fluidml_b200.executor import Executor


def logits_fp64(model, x):
    """The graph as torch runs it in fp64 on the GPU, four images at a time."""
    consts = {k: torch.from_numpy(v).cuda().double() for k, v in model.initializers.items() if v.dtype == np.float32}
    out = []
    for part in torch.from_numpy(x).split(4):
        v = {"input": part.cuda().double()}
        for n in model.nodes:
            a = [consts[i] if i in consts else v[i] for i in n.inputs]
            if n.op_type == "Conv":
                r = torch.nn.functional.conv2d(*a, padding=1)
            elif n.op_type == "MaxPool":
                r = torch.nn.functional.max_pool2d(a[0], 2)
            elif n.op_type == "Gemm":
                r = a[0] @ a[1].T + a[2]
            else:
                r = {"Relu": torch.relu, "Flatten": lambda t: t.flatten(1)}[n.op_type](a[0])
            v[n.outputs[0]] = r
        out.append(r.cpu().numpy())
    return np.concatenate(out)


@pytest.mark.parametrize("batch,tolerance", [(1, 5e-5), (32, 1.7e-4)])
def test_logits(batch, tolerance):
    """Relative error (2-norm); measured 2.5e-5 and 1.11e-4.  (3xTF32 contractions, whose parts are truncated
    and summed 8 at a time: 6.5e-5 and 2.5e-4.)"""
    model, x = models.build_vgg16(batch=batch), models.vgg_inputs(batch=batch)
    y = {"output": np.zeros((batch, 1000), np.float32)}
    Executor.make_dp_greedy("v").compile(model.to_bytes()).invoke({**x, **y})
    ref = logits_fp64(model, x["input"])
    assert np.linalg.norm(y["output"] - ref) <= tolerance * np.linalg.norm(ref)

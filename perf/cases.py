"""Workloads of the executor: what a program that serves models with it has it do.

A case is one model at one input shape.  A pass is one `Executor.invoke`, the call a serving
program makes per request: host arrays in (copied to the device), the whole forward pass, host
arrays out.  The compiled executor is what such a program keeps between requests, so it is built
once per model and shape and every request of that shape goes through it; a seed stands for
another request (other token ids, another padding of the batch, other images).

Weights are the seeded ones of `fluidml_b200.models`.  `pinned` cases hand over page-locked
arrays (`pinned_empty`), as a server does that owns its request buffers; the others hand over
ordinary numpy arrays, as a script does.
"""
from __future__ import annotations

import math

import numpy as np

from fluidml_b200 import models
from fluidml_b200.executor import Executor, pinned_empty

VOCAB = 30522       # of the encoders
NEOX_VOCAB = 50304  # of the decoder

# (layers, hidden, heads, ffn): the full-size encoder, its halved depth, and the small ones used
# where latency or cost rules out the full size
_ENCODERS = ((2, 128, 2, 512), (4, 256, 4, 1024), (4, 512, 8, 2048), (6, 768, 12, 3072), (12, 768, 12, 3072))
_CONVBERTS = ((4, 256, 8, 1024), (6, 768, 12, 3072), (12, 768, 12, 3072))
_DECODERS = ((4, 256, 4, 1024), (6, 512, 8, 2048), (12, 1024, 16, 4096), (24, 1024, 16, 4096))


def _tokens(name, model, size, batch, seq, pinned, mode="dp_greedy"):
    layers, hidden, heads, ffn = size
    return {"name": name, "model": model, "layers": layers, "hidden": hidden, "heads": heads, "ffn": ffn,
            "batch": batch, "seq": seq, "pinned": pinned, "mode": mode}


def _images(name, model, batch, image, pinned, mode="dp_greedy"):
    return {"name": name, "model": model, "batch": batch, "image": image, "pinned": pinned, "mode": mode}


def listed():
    return [
        # the smallest call: one short sentence through a two-layer encoder, default layouts
        _tokens("encoder_2l_b1_s16", "bert", _ENCODERS[0], 1, 16, False, "plain_greedy"),
        # the benchmark's headline: one sentence of 128 tokens, full-size encoder
        _tokens("bert_base_b1_s128", "bert", _ENCODERS[-1], 1, 128, True),
        # a few sentences of a length nobody tuned for, from ordinary arrays
        _tokens("bert_base_b3_s77", "bert", _ENCODERS[-1], 3, 77, False),
        # offline embedding of documents: a full batch of long ragged texts
        _tokens("bert_base_b16_s384", "bert", _ENCODERS[-1], 16, 384, True),
        # image classification, one picture per request and in batches
        _images("vgg16_b1", "vgg16", 1, 224, False),
        _images("vgg16_b32", "vgg16", 32, 224, True),
        _images("efficientnet_b0_b1", "efficientnet_b0", 1, 224, True),
        _images("efficientnet_b0_b5_i192", "efficientnet_b0", 5, 192, False),
        _images("efficientnet_b0_b64", "efficientnet_b0", 64, 224, True),
        # the mixed attention / span-convolution encoder at its benchmark shape
        _tokens("convbert_base_b8_s128", "convbert", _CONVBERTS[-1], 8, 128, True),
        # decoder prefill: one short odd prompt, and the benchmark's four prompts of 512 tokens
        _tokens("gpt_neox_b1_s77", "gpt_neox", _DECODERS[-1], 1, 77, False),
        _tokens("gpt_neox_b4_s512", "gpt_neox", _DECODERS[-1], 4, 512, True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the five models, any size of it, batch and length (or image side)
    spread over their logarithm, capped at the largest listed amount of work."""
    model = rng.choice(("bert", "bert", "vgg16", "efficientnet_b0", "convbert", "gpt_neox"))
    pinned = rng.random() < 0.5
    mode = "plain_greedy" if rng.random() < 0.15 else "dp_greedy"
    if model == "vgg16":
        image = 32 * rng.randint(4, 8)
        c = _images("", model, _log_int(rng, 1, 32 * 224 * 224 // (image * image) or 1), image, pinned, mode)
    elif model == "efficientnet_b0":
        image = 32 * rng.randint(4, 9)
        c = _images("", model, _log_int(rng, 1, 64 * 224 * 224 // (image * image)), image, pinned, mode)
    else:
        sizes, most, longest = {"bert": (_ENCODERS, 6144, 512), "convbert": (_CONVBERTS, 2048, 384),
                                "gpt_neox": (_DECODERS, 2048, 512)}[model]
        seq = _log_int(rng, 12, longest)
        batch = _log_int(rng, 1, max(1, min(48, most // seq)))
        c = _tokens("", model, rng.choice(sizes), batch, seq, pinned, mode)
    del c["name"]
    return c


# ------------------------------------------------------------------ executors and requests
_MAKE = {"dp_greedy": Executor.make_dp_greedy, "plain_greedy": Executor.make_plain_greedy}
_EXECUTORS = {}  # compiled executors by model and shape, kept as a serving program keeps them


def _build(case):
    if case["model"] == "vgg16":
        return models.build_vgg16(batch=case["batch"], image=case["image"])
    if case["model"] == "efficientnet_b0":
        # std 0.16: at 0.02 the logits of a batch-norm-free network are all bias
        return models.build_efficientnet_b0(batch=case["batch"], image=case["image"], std=0.16)
    build = {"bert": models.build_bert, "convbert": models.build_convbert, "gpt_neox": models.build_gpt_neox}[case["model"]]
    return build(**{k: case[k] for k in ("layers", "hidden", "heads", "ffn", "batch", "seq")})


def _executor(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "pinned")))
    if key not in _EXECUTORS:
        model = _build(case)
        outputs = [(o.name, tuple(o.shape)) for o in model.outputs]
        _EXECUTORS[key] = (_MAKE[case["mode"]](case["model"]).compile(model.to_bytes()), outputs)
    return _EXECUTORS[key]


def _request(case, seed):
    """What one request brings: images ~ N(0, 1), or token ids with, for the encoders, the mask of
    a batch that is padded to its longest text (half full at the least)."""
    rng = np.random.default_rng(seed)
    b = case["batch"]
    if "image" in case:
        return {"input": rng.standard_normal((b, 3, case["image"], case["image"]), dtype=np.float32)}
    s = case["seq"]
    if case["model"] == "gpt_neox":
        return {"input_ids": rng.integers(0, NEOX_VOCAB, (b, s), dtype=np.int64)}
    lengths = rng.integers((s + 1) // 2, s + 1, b)
    lengths[rng.integers(0, b)] = s
    return {"input_ids": rng.integers(0, VOCAB, (b, s), dtype=np.int64),
            "attention_mask": (np.arange(s)[None, :] < lengths[:, None]).astype(np.float32)}


def prepare(case, seed):
    executor, outputs = _executor(case)
    empty = pinned_empty if case["pinned"] else np.empty
    args = {}
    for name, value in _request(case, seed).items():
        args[name] = empty(value.shape, value.dtype)
        args[name][...] = value
    results = {}
    for name, shape in outputs:
        results[name] = args[name] = empty(shape, np.float32)
    return {"executor": executor, "args": args, "results": results}


def run(state):
    state["executor"].invoke(state["args"])
    return state["results"]


# ------------------------------------------------------------------ work and tolerance
def _token_work(c):
    """(multiply-adds, weight floats, input and output bytes) of a transformer pass."""
    layers, h, f, b, s = c["layers"], c["hidden"], c["ffn"], c["batch"], c["seq"]
    tokens = b * s
    io = tokens * 8 + tokens * h * 4
    gathered = tokens * h  # embedding rows
    attention = 2 * tokens * s * h  # scores and context
    if c["model"] == "gpt_neox":  # causal: a query sees half of the keys
        per_layer = 4 * h * h + 2 * h * f
        return layers * (tokens * per_layer + attention // 2), layers * per_layer + gathered, io
    io += tokens * 4
    gathered += s * h  # position rows
    if c["model"] == "bert":
        per_layer = 4 * h * h + 2 * h * f
        macs, floats = layers * (tokens * per_layer + attention) + b * h * h, layers * per_layer + h * h
        return macs, floats + gathered, io + b * h * 4
    heads = c["heads"] // 2
    w = h // 2  # width of either branch
    per_layer = 5 * h * w + 9 * h + w * heads * 9 + h * h + 2 * h * f
    span = tokens * w * 9  # the dynamic window
    return layers * (tokens * per_layer + attention // 2 + span), layers * per_layer + gathered, io


def _vgg_work(c):
    macs = floats = 0
    cin, side = 3, c["image"]
    for width in (64, 64, "M", 128, 128, "M", 256, 256, 256, "M", 512, 512, 512, "M", 512, 512, 512, "M"):
        if width == "M":
            side //= 2
            continue
        macs += c["batch"] * side * side * width * cin * 9
        floats += width * cin * 9
        cin = width
    for n, k in ((4096, 512 * side * side), (4096, 4096), (1000, 4096)):
        macs += c["batch"] * n * k
        floats += n * k
    return macs, floats, 4 * c["batch"] * (3 * c["image"] ** 2 + 1000)


def _efficientnet_work(c):
    macs = floats = 0
    b, side, cin = c["batch"], c["image"] // 2, 32

    def conv(n, k, out_side):
        nonlocal macs, floats
        macs += b * out_side * out_side * n * k
        floats += n * k

    conv(32, 27, side)
    for expand, kernel, stride, cout, repeats in ((1, 3, 1, 16, 1), (6, 3, 2, 24, 2), (6, 5, 2, 40, 2), (6, 3, 2, 80, 3),
                                                  (6, 5, 1, 112, 3), (6, 5, 2, 192, 4), (6, 3, 1, 320, 1)):
        for r in range(repeats):
            mid = cin * expand
            if expand != 1:
                conv(mid, cin, side)
            side = -(-side // (stride if r == 0 else 1))
            conv(mid, kernel * kernel, side)
            conv(max(1, cin // 4), mid, 1)
            conv(mid, max(1, cin // 4), 1)
            conv(cout, mid, side)
            cin = cout
    conv(1280, cin, side)
    conv(1000, 1280, 1)
    return macs, floats, 4 * b * (3 * c["image"] ** 2 + 1000)


def work(case):
    """Contractions of the model (two operations per multiply-add), every weight read once, the
    request read once and the result written once; activations need not leave the chip."""
    count = {"vgg16": _vgg_work, "efficientnet_b0": _efficientnet_work}.get(case["model"], _token_work)
    macs, floats, io = count(case)
    return {"bytes": 4 * floats + io, "flops": 2 * macs}


def tolerance(case):
    """fp32 in and out, fp32-accurate contractions.  The tensor cores' accumulators truncate, so a
    contraction is off by about 1e-5 and a whole network by 5e-6 to 5e-5 against fp32 FMA; VGG-16's
    sums of up to 25,088 products of one sign (ReLU inputs) bring its logits to 6e-5 to 2.5e-4."""
    return {"rel": 5e-4, "max": 5e-3} if case["model"] == "vgg16" else {"rel": 1e-4, "max": 2e-3}

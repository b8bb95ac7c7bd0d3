"""The work that users have this engine do, as cases that can be timed.

A case is one call (or one decode) through the public Python API on one of the repository's own model shapes:

  entry    how the caller holds its data
             predict        one sample in an ordinary host array, `Model.predict`: the answer to one request
             multi          a list of separately allocated host samples, `Model.predict_multi`
             batch          one host array of samples, `Model.predict_batch`
             device         a batch that is already on the GPU, `Model.predict_batch_device` on the caller's stream
             generate       greedy decoding: prompts go in token by token, then every choice is fed back
             score          decoding with given tokens (a prompt, a text to be rated): the logits of every position are read
  bytes    images arrive as bytes and become floats on the GPU (`bytes_range`)
  pinned   the host array lies in page-locked memory

Models are loaded once and kept, as a program that serves keeps them; decode sessions too (`reset` starts the next
batch of sequences).  The weights are seeded and do not depend on a case's seed; every input does.
"""
import functools
import json
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "frugally-deep_b200"))  # the package of the tree that is the working folder

import fdeep_b200  # noqa: E402
from fdeep_b200 import model_writer as mw  # noqa: E402

# Decoders: the reduced shape of bench.py, and blocks as wide as GPT-2 small's (4 of its 12, a vocabulary that keeps the
# model text small enough to be written in seconds; a position runs the same chain of products per block).
DECODERS = {
    "decoder256": dict(vocab=4099, ctx=256, dim=256, layers=4, heads=4, ffn=1024),
    "decoder768": dict(vocab=4099, ctx=256, dim=768, layers=4, heads=12, ffn=3072),
}
LSTM = dict(vocab=20000, dim=128, units=512)
MOBILENET_SIZES = (96, 128, 160, 192, 224)


def listed():
    return [
        # one thumbnail, one answer: the smallest request there is, all latency
        dict(name="cnn: one image", model="cnn", entry="predict", n=1, size=32, bytes=False),
        # a shard of a data set of thumbnails, as decoded from image files
        dict(name="cnn: 1024 byte images", model="cnn", entry="batch", n=1024, size=32, bytes=True, pinned=False),
        # interactive classification of one photo
        dict(name="resnet50: one image", model="resnet50", entry="predict", n=1, size=224, bytes=False),
        # what a request queue gives: an odd number of photos, each in memory of its own, as bytes
        dict(name="resnet50: 37 byte images", model="resnet50", entry="multi", n=37, size=224, bytes=True),
        # the benchmark's batch, produced on the GPU by an earlier stage
        dict(name="resnet50: 256 on the GPU", model="resnet50", entry="device", n=256, size=224),
        # a few frames of a camera on a small network
        dict(name="mobilenetv2: 5 on the GPU", model="mobilenetv2", entry="device", n=5, size=160),
        # offline classification of a large set, float images from page-locked host memory
        dict(name="mobilenetv2: 384 images", model="mobilenetv2", entry="batch", n=384, size=224, bytes=False, pinned=True),
        # three short texts of one request: the time steps follow one another whatever the batch
        dict(name="lstm: 3 texts of 120", model="lstm", entry="multi", n=3, steps=120),
        # the benchmark's batch of texts
        dict(name="lstm: 4096 texts of 200", model="lstm", entry="device", n=4096, steps=200),
        # two users of a small decoder
        dict(name="decode: 2 sequences", model="decoder256", entry="generate", n=2, prompt=16, new=48),
        # a full batch of sequences, the benchmark's prompt
        dict(name="decode: 64 sequences", model="decoder768", entry="generate", n=64, prompt=32, new=32),
        # rating given texts: every token is known, every position's logits are read
        dict(name="decode: 19 given texts", model="decoder768", entry="score", n=19, prompt=80, new=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["cnn", "resnet50", "mobilenetv2", "lstm", "decoder256", "decoder768"])
    if model in DECODERS:
        prompt = rng.randint(4, 80)
        if rng.random() < 0.4:
            return dict(model=model, entry="score", n=_log(rng, 1, 64), prompt=prompt, new=0)
        return dict(model=model, entry="generate", n=_log(rng, 1, 64), prompt=prompt, new=rng.randint(4, 48))
    entry = rng.choice(["predict", "multi", "batch", "device", "device"])
    most = dict(cnn=2048, resnet50=256, mobilenetv2=384, lstm=4096)[model]
    n = 1 if entry == "predict" else _log(rng, 2, most)
    if entry == "multi":
        n = min(n, 128)
    case = dict(model=model, entry=entry, n=n)
    if model == "lstm":
        case["steps"] = rng.randint(20, 200)
        return case
    case["size"] = 32 if model == "cnn" else 224 if model == "resnet50" else rng.choice(MOBILENET_SIZES)
    if entry != "device":
        case["bytes"] = rng.random() < 0.5
    if entry == "batch":
        case["pinned"] = rng.random() < 0.5
    return case


# ---- what a program keeps: models and sessions -------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _model(name, size=0, first=False):
    if name == "cnn":
        js = mw.build_small_cnn(size=size)
    elif name == "resnet50":
        js = mw.build_resnet50(size=size, top="linear")  # the softmax of random weights saturates: logits tell more
    elif name == "mobilenetv2":
        js = mw.build_mobilenetv2(size=size)
    elif name == "lstm":
        js = mw.build_text_lstm(seq_len=None, **LSTM)    # texts of any length
    else:
        js = mw.build_gpt2_step(first=first, **DECODERS[name])
    text = json.dumps(js, allow_nan=False, separators=(",", ":"))
    return fdeep_b200.read_model_from_string(text, verify=False, devices=[0], skinny_products=name in DECODERS)


@functools.lru_cache(maxsize=4)
def _session(name, n, positions):
    return fdeep_b200.DecodeSession(_model(name, first=True), _model(name, first=False), batch=n, max_len=positions)


def _sample_shape(case):
    return [case["steps"]] if case["model"] == "lstm" else [case["size"], case["size"], 3]


def _positions(case):
    # the last token that is chosen is not fed back
    return case["prompt"] + max(case["new"] - 1, 0)


def _inputs(case, seed):
    """The case's samples as one GPU tensor, made from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    shape = [case["n"]] + _sample_shape(case)
    if case["model"] == "lstm":
        return torch.randint(1, LSTM["vocab"], shape, generator=g, device="cuda").float()
    if case.get("bytes"):
        return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)
    if case["model"] == "cnn":
        return torch.rand(shape, generator=g, device="cuda")
    if case["model"] == "mobilenetv2":
        return torch.rand(shape, generator=g, device="cuda") * 2 - 1
    return torch.randn(shape, generator=g, device="cuda")


def prepare(case, seed):
    name, entry = case["model"], case["entry"]
    if name in DECODERS:
        rng = np.random.default_rng(int(seed))
        tokens = rng.integers(0, DECODERS[name]["vocab"], size=(case["prompt"], case["n"])).astype(np.float32)
        return dict(case=case, tokens=tokens, session=_session(name, case["n"], _positions(case)))
    state = dict(case=case, model=_model(name, case.get("size", 0)))
    x = _inputs(case, seed)
    if entry == "device":
        shape = _sample_shape(case)
        out_shape = state["model"].infer_shapes([shape])[0]
        state.update(x=x, shape=shape, out=torch.empty([case["n"]] + out_shape, device="cuda"), stream=torch.cuda.Stream())
        torch.cuda.synchronize()
        return state
    host = x.cpu()
    if case.get("pinned"):
        host = host.pin_memory()
    state["x"] = host.numpy()
    if entry != "batch":
        state["samples"] = [[np.array(s)] for s in state["x"]]  # each in memory of its own
    return state


def run(state):
    case = state["case"]
    entry = case["entry"]
    span = (0.0, 1.0) if case.get("bytes") else None
    if entry == "predict":
        return state["model"].predict_multi(state["samples"], bytes_range=span)[0] if span else state["model"].predict(state["samples"][0])
    if entry == "multi":
        return np.stack([o[0] for o in state["model"].predict_multi(state["samples"], bytes_range=span)])
    if entry == "batch":
        return state["model"].predict_batch([state["x"]], bytes_range=span)
    if entry == "device":
        state["model"].predict_batch_device([state["x"].data_ptr()], [state["shape"]], case["n"], [state["out"].data_ptr()],
                                            stream=state["stream"].cuda_stream)
        return state["out"]
    session, tokens = state["session"], state["tokens"]
    session.reset()
    if entry == "score":
        return np.stack([session.step(t, want_logits=True)[1] for t in tokens])
    chosen = []
    for pos in range(_positions(case)):
        nxt, _ = session.step(tokens[pos] if pos < case["prompt"] else None)
        if pos >= case["prompt"] - 1:
            chosen.append(nxt)
    return np.stack(chosen).astype(np.int64)


# ---- what a pass cannot do without -------------------------------------------------------------------------
#: parameters of the image models, and multiply-adds of one image of side 224 (they grow with the square of the side)
_IMAGE_MODELS = {"cnn": (3 * 288 + 32 + 288 * 64 + 64 * 5 + 64 * 128 + 128 + 1290, None),
                 "resnet50": (25.6e6, 3.858e9), "mobilenetv2": (3.5e6, 0.3008e9)}


def work(case):
    n = case["n"]
    if case["model"] in DECODERS:
        c = DECODERS[case["model"]]
        d, positions = c["dim"], _positions(case)
        weights = c["layers"] * (4 * d * d + 2 * d * c["ffn"]) + d * c["vocab"]
        # every position depends on the one before, so it meets all weights anew, and the keys and values of the rows so far
        rows = 2 * c["layers"] * d * n * positions * (positions + 1) / 2
        logits = n * c["vocab"] * positions if case["entry"] == "score" else n * case["new"]
        return {"bytes": 4.0 * (weights * positions + rows + logits), "flops": 2.0 * weights * n * positions + 2.0 * rows}
    if case["model"] == "lstm":
        dim, units, steps = LSTM["dim"], LSTM["units"], case["steps"]
        macs = steps * 4 * units * (dim + 3 * units)
        params = 4 * units * (dim + 3 * units + 2) + LSTM["vocab"] * dim
        return {"bytes": 4.0 * (params + n * (steps + 1)), "flops": 2.0 * macs * n}
    params, macs = _IMAGE_MODELS[case["model"]]
    side = case["size"]
    if macs is None:
        macs = side * side * 27 * 32 + (side // 2) ** 2 * 288 * 64 + 64 * 128 + 1280
    else:
        macs *= (side / 224.0) ** 2
    outputs = 10 if case["model"] == "cnn" else 1000
    return {"bytes": 4.0 * (params + n * outputs) + n * side * side * 3 * (1 if case.get("bytes") else 4), "flops": 2.0 * macs * n}


def tolerance(case):
    if case["entry"] == "generate":
        # token numbers: two logits nearer to one another than their rounding errors may be taken either way round
        return {"differ": 0.01}
    # fp32 all the way: sums of up to 4608 products rounded in another order, through up to 50 layers (or 200 time steps)
    # that pass the error on; values near zero are held against the output's root mean square
    return {"rel": 3e-5, "max": 3e-4} if case["model"] in ("resnet50", "mobilenetv2") else {"rel": 1e-5, "max": 1e-4}

"""Performance cases: the work a program gives this framework, through its public entry points.

A case names a model shape of `synth.SHAPES`, a weight format, and one of the four things programs do with a model:

  step    one token of one stream: Model.run(id), logits to the host (the chat loop, the benchmark driver)
  serve   one token of each of `streams` streams: Model.decode, then the next ids: the arg-max that comes with it, or,
          with "sampled", Model.sample over the logits that stay on the device
  greedy  `tokens` greedy tokens of `streams` streams without a host round trip: Model.decode_greedy
  prompt  `tokens` tokens of one stream at once: Model.run(ids), last logits to the host

Weights are random with the distributions of `synth.device_tensors`, drawn from the seed; the model is what such a
program keeps.  A pass continues from the state the pass before it left, as a conversation does.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

frb = importlib.import_module("faster-rwkv_b200")

# A trained model's logits spread a few times wider than unit-variance random ones: a sampler that met those would keep
# thousands of almost equal candidates.
HEAD_GAIN = 4.0

STEP_SHAPES = ("c0", "c1", "c3", "c4")
SERVE_SHAPES = ("c0", "c1", "c3")
FORMATS = ("fp16", "int8", "int4")
MAX_STREAMS = 256
MAX_PROMPT = 4096


def listed():
    return [
        # one user at a time: the chat loop and the benchmark driver call run(id) once per token.  The smallest model,
        # where a token is short and every fixed cost shows ...
        {"name": "step_c0_fp16", "kind": "step", "shape": "c0", "weights": "fp16"},
        # ... the ordinary one, in the format of a converted file and in the smallest one ...
        {"name": "step_c1_fp16", "kind": "step", "shape": "c1", "weights": "fp16"},
        {"name": "step_c1_int4", "kind": "step", "shape": "c1", "weights": "int4"},
        # ... the newer architecture, with its per-head state matrices ...
        {"name": "step_c3_fp16", "kind": "step", "shape": "c3", "weights": "fp16"},
        # ... and the largest model, quantised as its users run it
        {"name": "step_c4_int8", "kind": "step", "shape": "c4", "weights": "int8"},
        # a handful of conversations on one device
        {"name": "serve_3_c1_int4", "kind": "serve", "shape": "c1", "weights": "int4", "streams": 3, "sampled": False},
        # a small server: every stream samples its next token with temperature and top-p
        {"name": "serve_16_c1_int8", "kind": "serve", "shape": "c1", "weights": "int8", "streams": 16, "sampled": True},
        # a busy server, the number of streams as it happens to be
        {"name": "serve_100_c1_fp16", "kind": "serve", "shape": "c1", "weights": "fp16", "streams": 100, "sampled": False},
        # offline generation with the device full: the benchmark's own workload
        {"name": "greedy_256_c1_int4", "kind": "greedy", "shape": "c1", "weights": "int4", "streams": 256, "tokens": 8},
        # a user's message, a document, and the longest prompt of the benchmark
        {"name": "prompt_29_c1_int4", "kind": "prompt", "shape": "c1", "weights": "int4", "tokens": 29},
        {"name": "prompt_1000_c1_fp16", "kind": "prompt", "shape": "c1", "weights": "fp16", "tokens": 1000},
        {"name": "prompt_4096_c3_fp16", "kind": "prompt", "shape": "c3", "weights": "fp16", "tokens": 4096},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(("step", "serve", "serve", "serve", "greedy", "prompt", "prompt", "prompt"))
    if kind == "step":
        return {"kind": kind, "shape": rng.choice(STEP_SHAPES), "weights": rng.choice(FORMATS)}
    case = {"kind": kind, "shape": rng.choice(SERVE_SHAPES if kind != "greedy" else ("c0", "c1")), "weights": rng.choice(FORMATS)}
    if kind == "serve":
        case.update(streams=_log_int(rng, 2, MAX_STREAMS), sampled=rng.random() < 0.25)
    elif kind == "greedy":
        case.update(streams=_log_int(rng, 1, MAX_STREAMS), tokens=rng.randint(2, 8))
    else:
        case.update(tokens=_log_int(rng, 2, MAX_PROMPT))
    return case


def _streams(case):
    return case.get("streams", 1)


class _DeviceArray:
    """Device memory of a model as something torch.as_tensor takes without a copy; it keeps the model alive."""

    def __init__(self, model, ptr, shape, strides):
        self.model = model
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides, "typestr": "<f4", "version": 3}


def _logits(model, streams):
    """The logits that stay on the device, [streams, vocab] (fr_b200_logits_device)."""
    p = ctypes.c_void_p()
    lib = frb.lib()
    lib.fr_b200_logits_device.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_void_p)]
    frb.check(lib.fr_b200_logits_device(model.handle, ctypes.byref(p)), "fr_b200_logits_device")
    ld = lib.fr_b200_vocab_padded(model.handle)
    return torch.as_tensor(_DeviceArray(model, p.value, (streams, model.vocab), (ld * 4, 4)), device="cuda")


def _state(model, streams):
    """The recurrent state on the device, one [streams, layers, elements] tensor for each of the layer's fp32 state
    tensors (aa, bb, pp or the per-head matrices; fr_b200_state_tensor).  The token-shift states change place from token
    to token; the next pass's logits show them."""
    lib = frb.lib()
    count = lib.fr_b200_state_count(model.handle)

    def at(slot, layer, index):
        p, dt, n = ctypes.c_void_p(), ctypes.c_int(), ctypes.c_int64()
        frb.check(lib.fr_b200_state_tensor(model.handle, slot, layer, index, ctypes.byref(p), ctypes.byref(dt), ctypes.byref(n)),
                  "fr_b200_state_tensor")
        return p.value, n.value

    got = []
    layers = model.shape.n_layer
    for index in range(1, count - 1):
        p, n = at(0, 0, index)
        by_layer = at(0, 1, index)[0] - p
        by_slot = at(1, 0, index)[0] - p if streams > 1 else by_layer * layers
        assert at(streams - 1, layers - 1, index)[0] == p + by_slot * (streams - 1) + by_layer * (layers - 1)
        got.append(torch.as_tensor(_DeviceArray(model, p, (streams, layers, n), (by_slot, by_layer, 4)), device="cuda"))
    return got


def prepare(case, seed):
    shape = frb.synth.SHAPES[case["shape"]]
    weights, streams = case["weights"], _streams(case)
    gen = frb.synth.device_tensors(shape, seed, "cuda", "fp16" if weights == "fp16" else "fp32")
    tensors = ((n, t * HEAD_GAIN if n == "head.weight" else t) for n, t in gen)

    class Tensors:  # one tensor at a time on the device, as a loader hands them over
        def items(self):
            return tensors

    model = frb.Model(Tensors(), "cuda " + weights, max_batch=streams, shape=shape)
    rng = np.random.default_rng(seed)
    n = case["tokens"] if case["kind"] == "prompt" else streams
    return {"case": dict(case), "model": model, "ids": rng.integers(0, shape.vocab, n).astype(np.int32),
            "uniform": rng.random(streams).astype(np.float32),
            "logits": _logits(model, streams), "state": _state(model, streams)}


def run(state):
    case, model, ids = state["case"], state["model"], state["ids"]
    kind = case["kind"]
    if kind == "step":
        return {"logits": model.run(int(ids[0])), "state": state["state"]}
    if kind == "prompt":
        return {"logits": model.run(ids), "state": state["state"]}
    if kind == "greedy":
        return {"ids": model.decode_greedy(ids, case["tokens"])}
    if case["sampled"]:
        model.decode(ids, want_logits=False)
        picked = model.sample(len(ids), 1.0, 0, 0.8, state["uniform"])
    else:
        picked = model.decode(ids, want_logits=False, want_argmax=True)
    return {"ids": picked, "logits": state["logits"], "state": state["state"]}


def work(case):
    s = frb.synth.SHAPES[case["shape"]]
    C, F, L, V, H = s.n_embd, s.n_ffn, s.n_layer, s.vocab, s.n_head
    v5 = s.version.startswith("5")
    squares = 6 if s.version in ("5.1", "5.2") else 5
    layer_params = L * (squares * C * C + 2 * C * F)
    outputs = L * ((squares + 1) * C + F)   # output channels of all layers
    params = layer_params + C * V
    weights = {"fp16": 2.0 * params, "int8": params + 2.0 * (outputs + V), "int4": params / 2 + params / 16}[case["weights"]]
    act = 2 if case["weights"] == "fp16" else 4
    state = L * (2 * C * act + (H * 4096 * 4 if v5 else 3 * C * 4))
    streams, kind = _streams(case), case["kind"]
    if kind == "prompt":
        T = case["tokens"]
        emb = T * C * act
        flops = 2.0 * T * layer_params + 2.0 * C * V + (T * L * 6.0 * C * 64 if v5 else 0.0)
        return {"bytes": weights + emb + 2 * state + V * 4, "flops": flops}
    steps = case["tokens"] if kind == "greedy" else 1
    flops = streams * (2.0 * params + (L * 6.0 * C * 64 if v5 else 0.0))
    step_bytes = weights + streams * (C * act + 2 * state + (0 if kind == "greedy" else V * 4))
    return {"bytes": steps * step_bytes, "flops": steps * flops}


def tolerance(case):
    # prompts multiply fp16 activations, one token per stream uses fp16 pairs and hands vectors on with 16 significant
    # bits; the shift states are fp16 in fp16 models.  Picked ids differ where two candidates are closer than that.
    if case["kind"] == "prompt":
        return {"rel": 2e-3}
    if case["kind"] == "step":
        return {"rel": 1e-3}
    return {"rel": 1e-3, "differ": 0.01}

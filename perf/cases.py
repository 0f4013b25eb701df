"""The work that a user of this framework has it do, as cases that can be timed.

A case names an entry point (`kind`), one of the model configurations of `ullis_b200.synth` where the entry point takes
a model, and the sizes of the call.  `gain_one` chooses between the two weight distributions of the benchmark
configurations: LayerNorm gain 1 + N(0, 0.02), what a model in training has (no channel of Q, K or V is constant), and
N(0, 0.02), the one the headline configuration states (about half of the channels are constant).

Everything goes through the host-array interface (`CudaRuntime`, `CudaHeron`, `CudaGenerateState`, `CudaTrainState`):
token ids, activations and bit planes come from host memory and the results end in host memory.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ullis_b200 import cuda, synth

IGNORE = cuda.CE_NO_IGNORE
LEARNING_RATE = 0.005


def listed():
    return [
        # one short sequence of the small model scored: what a user tries first; launches and latency
        {"name": "score small, one sequence", "kind": "score", "model": "small", "gain_one": False, "batch": 1, "time": 512},
        # one full context of the default model: perplexity of a document
        {"name": "score default, one sequence", "kind": "score", "model": "default", "gain_one": False, "batch": 1,
         "time": 2048},
        # the headline workload: 64 full contexts
        {"name": "score default, 64 sequences", "kind": "score", "model": "default", "gain_one": False, "batch": 64,
         "time": 2048},
        # an evaluation batch of a model in training
        {"name": "score default in training, 16", "kind": "score", "model": "default", "gain_one": True, "batch": 16,
         "time": 2048},
        # an evaluation batch cut to an odd length
        {"name": "score default, ragged", "kind": "score", "model": "default", "gain_one": True, "batch": 5, "time": 1531},
        # the distribution over the next token at every position of a few prompts
        {"name": "logits small", "kind": "logits", "model": "small", "gain_one": True, "batch": 3, "time": 333},
        # a reply: a prompt fed token by token, then new tokens
        {"name": "generate, one sequence", "kind": "generate", "model": "default", "gain_one": True, "batch": 1,
         "prompt": 320, "new": 40},
        # many replies side by side
        {"name": "generate, 64 sequences", "kind": "generate", "model": "default", "gain_one": True, "batch": 64,
         "prompt": 96, "new": 32},
        # optimiser steps on fresh batches and the weights a checkpoint takes
        {"name": "train default", "kind": "train", "model": "default", "gain_one": True, "batch": 8, "time": 2048, "steps": 2},
        # the packed linear by itself (feed-forward width of the default model)
        {"name": "binary linear", "kind": "linear", "rows": 2048, "in": 512, "out": 2048},
        # the 1-bit attention by itself over long periodic streams
        {"name": "rosa standalone", "kind": "rosa", "batch": 8, "time": 8192, "channels": 512, "periodic": True},
        # one attention block at the size of a latency test
        {"name": "rosa block, one window", "kind": "block", "batch": 1, "time": 32, "channels": 256},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["score", "score", "score", "logits", "generate", "generate", "train", "linear", "rosa", "block"])
    gain_one = rng.random() < 0.6
    if kind == "linear":
        k, n = rng.choice([(256, 256), (256, 1024), (512, 512), (512, 2048), (512, 8192)])
        return {"kind": kind, "rows": _log(rng, 1, 4096 if n <= 2048 else 2048), "in": k, "out": n}
    if kind == "block":
        return {"kind": kind, "batch": rng.randint(1, 4), "time": _log(rng, 16, 2048), "channels": rng.choice([64, 256, 512])}
    if kind == "rosa":
        time = _log(rng, 64, 8192)
        channels = rng.choice([64, 256, 512])
        most = max(1, min(64, (8 * 8192 * 512) // (time * channels)))
        return {"kind": kind, "batch": _log(rng, 1, most), "time": time, "channels": channels, "periodic": rng.random() < 0.5}
    if kind == "generate":
        batch, new = _log(rng, 1, 64), rng.randint(8, 48)
        prompt = _log(rng, 16, 700 if batch <= 4 else 320 if batch <= 16 else 96)
        return {"kind": kind, "model": "default", "gain_one": gain_one, "batch": batch, "prompt": prompt, "new": new}
    if kind == "train":
        model = rng.choice(["small", "default"])
        return {"kind": kind, "model": model, "gain_one": True, "batch": rng.randint(1, 8),
                "time": _log(rng, 64, synth.CONFIGS[model][3]), "steps": 2}
    if kind == "logits":
        model = rng.choice(["tiny", "small", "default"])
        time = _log(rng, 8, synth.CONFIGS[model][3])
        return {"kind": kind, "model": model, "gain_one": gain_one, "batch": max(1, min(8, _log(rng, 1, 16), 4096 // time)),
                "time": time}
    model = rng.choice(["small", "default", "default"])
    time = _log(rng, 32, synth.CONFIGS[model][3])
    most = 64 if not gain_one or model == "small" else 16
    return {"kind": kind, "model": model, "gain_one": gain_one, "batch": _log(rng, 1, most), "time": time}


# ---- what a program keeps: the device's runtime, checkpoints and loaded models


@functools.lru_cache(maxsize=None)
def _runtime():
    return cuda.CudaRuntime(0)


@functools.lru_cache(maxsize=None)
def _checkpoint(model, gain_one):
    return synth.heron_checkpoint(model, batch_size=64, ln_gain_one=gain_one)


@functools.lru_cache(maxsize=None)
def _model(model, gain_one):
    return cuda.CudaHeron(_runtime(), _checkpoint(model, gain_one))


def _tokens(rng, vocab, shape):
    """Zipf(1.1) ids, the token distribution of the benchmark."""
    cdf = np.cumsum(np.arange(1, vocab + 1, dtype=np.float64) ** -1.1)
    return np.minimum(np.searchsorted(cdf / cdf[-1], rng.random(shape), side="right"), vocab - 1).astype(np.uint32)


def _f16(x):
    return synth.f16_bits(x)


def _words(rng, bits):
    w = rng.integers(0, 1 << 32, (bits + 31) // 32, dtype=np.uint32)
    if bits % 32:
        w[-1] &= np.uint32((1 << bits % 32) - 1)
    return w


def _packed(rng, out, inn):
    return {"bits": _words(rng, out * inn), "scale": _f16(rng.uniform(0.005, 0.02, out)),
            "bias": _f16(0.01 * rng.standard_normal(out))}


def _periodic_planes(seed, batch, time, channels):
    """Packed [B,T,C] planes of q, k, v: per stream a random period of 16..256, q and k from one base pattern, 10 % flips."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    period = torch.randint(16, 257, (batch, 1, channels), generator=g, device="cuda")
    phase = torch.arange(time, device="cuda").reshape(1, time, 1) % period
    qk, v = (torch.randint(0, 2, (batch, 256, channels), generator=g, device="cuda", dtype=torch.uint8) for _ in range(2))
    weight = 2 ** torch.arange(8, device="cuda", dtype=torch.int32)
    planes = []
    for base in (qk, qk, v):
        bits = torch.gather(base, 1, phase) ^ (torch.rand((batch, time, channels), generator=g, device="cuda") < 0.1)
        packed = (bits.reshape(-1, 8).to(torch.int32) * weight).sum(1).to(torch.uint8)
        planes.append(packed.cpu().numpy().view(np.uint32))
    return planes


def prepare(case, seed):
    rng = np.random.default_rng([seed, 0x5EED])
    kind = case["kind"]
    state = {"kind": kind, "case": case, "rt": _runtime()}
    if kind in ("score", "logits"):
        state["model"] = _model(case["model"], case["gain_one"])
        state["tokens"] = _tokens(rng, state["model"].vocab_size, case["batch"] * case["time"])
    elif kind == "generate":
        model = _model(case["model"], case["gain_one"])
        state["tokens"] = _tokens(rng, model.vocab_size, (case["prompt"] + case["new"], case["batch"]))
        state["generate"] = model.generate_state(case["batch"])
    elif kind == "train":
        model = cuda.CudaHeron(_runtime(), _checkpoint(case["model"], case["gain_one"]))
        state["tokens"] = _tokens(rng, model.vocab_size, (case["steps"], case["batch"] * case["time"]))
        state["model"], state["train"] = model, model.train_state()
    elif kind == "linear":
        state["x"] = rng.standard_normal(case["rows"] * case["in"], np.float32).astype(np.float16).astype(np.float32)
        state["w"] = _packed(rng, case["out"], case["in"])
    elif kind == "rosa":
        b, t, c = case["batch"], case["time"], case["channels"]
        state["planes"] = _periodic_planes(seed, b, t, c) if case["periodic"] else [_words(rng, b * t * c) for _ in range(3)]
        state["e"] = _f16(0.02 * rng.standard_normal(c))
    elif kind == "block":
        b, t, c = case["batch"], case["time"], case["channels"]
        state["x"] = rng.standard_normal(b * t * c, np.float32)
        state["p"] = {m: _f16(rng.uniform(0, 1, c)) for m in ("x_q", "x_k", "x_v")}
        state["p"].update({m: _packed(rng, c, c) for m in "qkvo"}, e=_f16(0.02 * rng.standard_normal(c)))
    return state


def _trained_tensors(model, train):
    """The weights a checkpoint of the trained model takes, FP16 as such and packed signs as words."""
    d, v, f = model.d_model, model.vocab_size, model.dim_ffn
    out = {"embedding": train.read("embedding", np.uint16, v * d).view(np.float16),
           "ln_out.weight": train.read("ln_out.weight", np.uint16, d).view(np.float16),
           "head.bits": train.read("head.bits", np.uint32, v * d // 32),
           "head.scale": train.read("head.scale", np.uint16, v).view(np.float16),
           "head.bias": train.read("head.bias", np.uint16, v).view(np.float16),
           "head.latent": train.read("head.latent", np.uint16, v * d).view(np.float16)}
    for i in range(model.n_layers):
        out[f"{i}.value"] = train.read(f"blocks.{i}.ffn.value", np.uint16, d * f).view(np.float16)
        out[f"{i}.key"] = train.read(f"blocks.{i}.ffn.key.bits", np.uint32, d * f // 32)
        out[f"{i}.o"] = train.read(f"blocks.{i}.rosa.o.bits", np.uint32, d * d // 32)
        out[f"{i}.e"] = train.read(f"blocks.{i}.rosa.e", np.uint16, d).view(np.float16)
    return out


def run(state):
    kind, case, rt = state["kind"], state["case"], state["rt"]
    if kind == "score":
        mean, loss_sum, n_valid, rows = state["model"].forward_ce(state["tokens"], state["tokens"], IGNORE, case["batch"],
                                                                  case["time"], want_row_loss=True)
        return {"mean": mean, "sum": loss_sum, "n_valid": n_valid, "rows": rows}
    if kind == "logits":
        return state["model"].logits(state["tokens"], case["batch"], case["time"])
    if kind == "generate":
        g = state["generate"]
        g.reset()
        for t in range(case["prompt"] - 1):
            g.step(state["tokens"][t])
        return [g.step(state["tokens"][t]) for t in range(case["prompt"] - 1, case["prompt"] + case["new"])]
    if kind == "train":
        losses = [state["train"].train_step(tokens, tokens, IGNORE, case["batch"], case["time"], LEARNING_RATE)["loss"]
                  for tokens in state["tokens"]]
        return {"losses": losses, **_trained_tensors(state["model"], state["train"])}
    if kind == "linear":
        w = state["w"]
        return rt.binary_linear(state["x"], w["bits"], w["scale"], w["bias"], case["rows"], case["in"], case["out"])
    if kind == "rosa":
        idx, out = rt.rosa_qkv_1bit_fwd(*state["planes"], state["e"], case["batch"], case["time"], case["channels"])
        return {"idx": idx, "out": out}
    return rt.rosa_block_forward(state["x"], state["p"], case["batch"], case["time"], case["channels"])


def _weights(model):
    """(bytes of the matrices a pass over the layers reads, multiply-adds per token of the layers, of the head)."""
    d, layers, vocab, _, f = synth.CONFIGS[model]
    layer_macs = 4 * d * d + 2 * d * f
    return layers * (4 * d * d // 8 + d * f // 8 + 2 * d * f) + vocab * d // 8, layers * layer_macs, d * vocab


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["rows"], case["in"], case["out"]
        return {"bytes": 4 * m * k + n * k // 8 + 4 * n + 4 * m * n, "flops": 2 * m * k * n}
    if kind in ("rosa", "block"):
        units = case["batch"] * case["time"] * case["channels"]
        if kind == "rosa":
            return {"bytes": units * (3 / 8 + 1 + 4), "flops": 0}
        c = case["channels"]
        return {"bytes": units * (4 + 3 / 8 + 1 + 4 + 4) + 4 * c * c // 8, "flops": 8 * units * c}
    d, layers, vocab, _, _ = synth.CONFIGS[case["model"]]
    weights, layer_macs, head_macs = _weights(case["model"])
    if kind == "generate":
        steps, batch = case["prompt"] + case["new"], case["batch"]
        # each step reads the weights and returns the logits of its tokens
        return {"bytes": steps * (weights + batch * (2 * d + 4 * vocab)), "flops": 2 * steps * batch * (layer_macs + head_macs)}
    rows = case["batch"] * case["time"]
    if kind == "train":
        # forward, and a gradient for the inputs and the weights of every linear but Q, K and V
        trained = layer_macs - 3 * layers * d * d + head_macs
        state = 6 * (vocab * d * 2 + layers * (d * d + 2 * d * synth.CONFIGS[case["model"]][4]))
        return {"bytes": case["steps"] * (8 * rows + 2 * state), "flops": case["steps"] * 2 * rows * (layer_macs + head_macs + 2 * trained)}
    out = 4 * rows * vocab if kind == "logits" else 4 * rows
    return {"bytes": weights + 2 * d * min(rows, vocab) + 4 * rows + out, "flops": 2 * rows * (layer_macs + head_macs)}


def tolerance(case):
    kind = case["kind"]
    if kind == "rosa":
        return "exact"                                  # indices, and +-e selected by them
    if kind == "generate":
        return {"rel": 1e-5}                            # f32 arithmetic in the reference's order
    if kind == "train":
        return {"rel": 5e-3, "max": 0.5, "differ": 5e-3}  # FP16 gradient operands; signs of latents near zero
    if kind == "logits":
        return {"rel": 2e-3}                            # FP16 operands, f32 accumulation, 2 to 12 layers
    return {"rel": 1e-3, "max": 2e-2, "differ": 0.0}    # FP16 operands, f32 accumulation

"""The work a user of this package has one GPU do, as cases that can be timed.

Three ways to use the package's models and operators, each through its public entry points:

  train    ``DDPTrainer.step`` / ``step_from_host``: one optimizer step of the data-parallel engine (examples/ddp_train.py, bench.py)
  loop     ``loss = model(tokens, targets); loss.backward()``: the forward and backward of a stock PyTorch loop, as under stock
           DistributedDataParallel (examples/stock_ddp.py), gradients gathered into one flat buffer as a one-bucket reduction needs them
  logits   ``model(tokens)`` without gradients: scoring / prefill

Models are the package's presets, and two cuts of the 1.3B family from bench/tp_bench.py.  Collectives between GPUs are not here: they
need peers, and one process on one GPU has none.
"""
import dataclasses
import math

import torch

from mccl_b200.models import build_decoder
from mccl_b200.models.decoder import PRESETS
from mccl_b200.parallel import DDPTrainer

#: name: (preset, what is changed, most tokens per pass of a drawn case)
_MODELS = {
    "tiny": ("tiny", {}, 4096),
    "70m": ("70m", {}, 16384),      # four times the headline batch of 16 x 256
    "110m": ("110m", {}, 8192),
    # RMSNorm / RoPE / SwiGLU, the benchmark's small model
    "swiglu": ("1.3b", {"vocab": 4096, "d_model": 1024, "n_layers": 4, "n_heads": 16, "d_ff": 4096, "max_seq": 1024}, 4096),
    # the widths of the 1.3B model with the twelve layers of one of two pipeline stages (bench/tp_bench.py --pp 2)
    "1.3b": ("1.3b", {"n_layers": 12}, 2048),
}


def _config(case):
    preset, changes, _ = _MODELS[case["model"]]
    return dataclasses.replace(PRESETS[preset], **changes)


def _case(name, kind, model, batch, seq, host=False):
    return {"name": name, "kind": kind, "model": model, "batch": batch, "seq": seq, "host": host}


def listed():
    return [
        # a unit-test sized model: nothing but launches and their gaps
        _case("train-tiny", "train", "tiny", 4, 64),
        # the headline benchmark, end to end: batch from pinned host memory, loss read back every step
        _case("train-70m", "train", "70m", 16, 256, host=True),
        # the same model with the batch somebody with 180 GB of memory would choose
        _case("train-70m-large", "train", "70m", 64, 256),
        # sequences that were not padded to a power of two
        _case("train-70m-ragged", "train", "70m", 8, 200),
        # the second headline model
        _case("train-110m", "train", "110m", 16, 256),
        # the RMSNorm / RoPE / SwiGLU family
        _case("train-swiglu", "train", "swiglu", 4, 1024),
        # stock training loops: small and uneven, and the headline shape
        _case("loop-tiny", "loop", "tiny", 8, 24),
        _case("loop-70m", "loop", "70m", 16, 256),
        # scoring: one short prompt, a full batch, a long uneven prompt on the large model
        _case("logits-70m-short", "logits", "70m", 1, 37),
        _case("logits-110m", "logits", "110m", 16, 256),
        _case("logits-1.3b", "logits", "1.3b", 1, 1537),
    ]


def _between(rng, low, high):
    """A whole number of [low, high], spread over the logarithm."""
    return min(high, max(low, round(low * (high / low) ** rng.random())))


def draw(rng):
    kind = rng.choice(("train", "train", "loop", "logits"))
    model = rng.choice(("tiny", "70m", "70m", "110m", "110m", "swiglu") + (("1.3b",) if kind == "logits" else ()))
    config, most = _config({"model": model}), _MODELS[model][2]
    seq = _between(rng, 16, config.max_seq)
    # whole blocks of 64 as often as not: batches are padded, prompts are not
    if rng.random() < 0.5:
        seq = max(64, seq // 64 * 64)
    # training the GELU models takes token counts in whole blocks of 64
    block = 64 if kind != "logits" and config.act == "gelu" else 1
    while block // math.gcd(seq, block) * seq > most:
        seq += 1
    unit = block // math.gcd(seq, block)
    batch = unit * _between(rng, 1, max(1, most // (seq * unit)))
    return {"kind": kind, "model": model, "batch": batch, "seq": seq, "host": kind == "train" and rng.random() < 0.5}


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    torch.manual_seed(seed)   # random-init weights
    preset, changes, _ = _MODELS[case["model"]]
    with dev:
        model = build_decoder(preset, **changes)
    g = torch.Generator().manual_seed(seed)
    ids = torch.randint(0, model.cfg.vocab, (case["batch"], case["seq"] + 1), generator=g)
    inp, tgt = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    if case["host"]:
        inp, tgt = inp.pin_memory(), tgt.pin_memory()
    else:
        inp, tgt = inp.to(dev), tgt.to(dev)
    state = {"kind": case["kind"], "host": case["host"], "model": model, "inp": inp, "tgt": tgt}
    if case["kind"] == "train":
        state["trainer"] = DDPTrainer(model, dev, lr=3e-4)
    elif case["kind"] == "loop":
        state["params"] = list(model.parameters())
        state["flat"] = torch.empty(sum(p.numel() for p in state["params"]), device=dev)
    return state


def run(state):
    if state["kind"] == "train":
        trainer = state["trainer"]
        step = trainer.step_from_host if state["host"] else trainer.step
        loss = step(state["inp"], state["tgt"])
        return {"loss": loss, "params": trainer.flat_p, "exp_avg": trainer.m, "exp_avg_sq": trainer.v}
    model = state["model"]
    if state["kind"] == "loop":
        model.zero_grad(set_to_none=True)
        loss = model(state["inp"], state["tgt"])
        loss.backward()
        torch.cat([p.grad.view(-1) for p in state["params"]], out=state["flat"])
        return {"loss": loss, "grads": state["flat"]}
    with torch.no_grad():
        return model(state["inp"])


def _sizes(case):
    """(parameters, multiply-adds per token of the matrix products, multiply-adds of causal attention in one forward)"""
    c = _config(case)
    tokens = case["batch"] * case["seq"]
    per_token = c.n_layers * (4 * c.d_model * c.d_model + (3 if c.act == "swiglu" else 2) * c.d_model * c.d_ff) + c.vocab * c.d_model
    attention = c.n_layers * tokens * case["seq"] * c.d_model   # two products, half of the square
    return c.param_count(), per_token, attention


def work(case):
    params, per_token, attention = _sizes(case)
    tokens = case["batch"] * case["seq"]
    forward = 2 * (per_token * tokens + attention)
    if case["kind"] == "train":   # fp32 parameters and both moments in and out
        return {"bytes": 24 * params + 16 * tokens, "flops": 3 * forward}
    if case["kind"] == "loop":    # fp32 parameters in, their gradients out
        return {"bytes": 8 * params + 16 * tokens, "flops": 3 * forward}
    vocab = _config(case).vocab
    return {"bytes": 4 * params + 8 * tokens + 2 * tokens * vocab, "flops": forward}


def tolerance(case):
    # bf16 activations and products all the way through a network of 2 to 16 layers, fp32 sums: the same model on stock PyTorch operators
    # in bf16 is 0.6e-2 to 2e-2 away as a whole.  Squared gradients (exp_avg_sq) carry twice the relative error of the gradients, and
    # gradients that are mostly cancellation (the key biases) differ by up to their own root mean square.
    if case["kind"] == "logits":
        return {"rel": 3e-2 if case["model"] == "1.3b" else 2e-2, "max": 0.3}
    return {"rel": 3e-2, "max": 0.95}

"""Performance cases: what a training or inference program of this framework spends its time on.

Four kinds of work, each through the calls that such a program makes:

* ``step``   -- one optimizer step of ``utils.TrainStep`` (captured in a CUDA graph): pinned tokens in, loss out.
* ``loop``   -- one optimizer step of the eager loop of the command line (``cli.train_main``): gradient accumulation over
  ``micro`` micro-batches, the loss read back after each, ``MixedPrecisionAdam`` with or without gradient clipping.
* ``logits`` -- a forward pass without gradients: what sampling runs for every new token, and an evaluation for a batch.
* ``layer``  -- forward and backward of one transformer block, gradients into the flat fp32 buffer: the unit that a
  pipeline stage or a larger model repeats.

Models are the presets of ``models`` (GPT-2 124M and XL, LLaMA-3 1B and 8B) with random weights and uniform random tokens.
"""
from __future__ import annotations

import copy
import dataclasses
import functools
import math

import torch

import tinyinfinitrain_b200 as tit
from tinyinfinitrain_b200.models import GPT2, GPT2_PRESETS, LLAMA3_PRESETS, LLaMA3
from tinyinfinitrain_b200.models.llama3 import LLaMA3Block
from tinyinfinitrain_b200.optim import FlatParams, MixedPrecisionAdam
from tinyinfinitrain_b200.utils import TrainStep

DEVICE = "cuda"
# the first steps of a learning-rate warm-up
LEARNING_RATE = 1e-6


def _case(name, do, model, dtype, batch, seq, micro=1, clip=0.0, layers=0):
    case = {"do": do, "model": model, "layers": layers, "dtype": dtype, "batch": batch, "seq": seq, "micro": micro,
            "clip": clip}
    return {"name": name, **case} if name else case


def listed():
    return [
        # one window of text generation at the command line's default batch and length: the window is run again for
        # every token, so latency and launches are what a user waits for
        _case("gpt2 sampling 4x64", "logits", "gpt2", "bf16", 4, 64),
        # validation: logits of a full batch
        _case("gpt2 evaluation 8x1024", "logits", "gpt2", "bf16", 8, 1024),
        # prompt of an odd length through the 1B model
        _case("llama3-1b prompt 1x1999", "logits", "llama3-1b", "bf16", 1, 1999),
        # the command line as it comes: eager bf16 loop at its default batch and length, accumulating twice
        _case("gpt2 loop 4x64", "loop", "gpt2", "bf16", 4, 64, micro=2),
        # the end-to-end check's setting: fp32, two micro-batches of 2 x 64
        _case("gpt2 fp32 loop 2x64", "loop", "gpt2", "fp32", 2, 64, micro=2),
        # fp32 training at a working size, with gradient clipping
        _case("gpt2 fp32 loop 4x512", "loop", "gpt2", "fp32", 4, 512, micro=1, clip=1.0),
        # fine-tuning on short texts: a small captured step
        _case("gpt2 step 2x128", "step", "gpt2", "bf16", 2, 128),
        # sequences of an odd length, odd batch
        _case("gpt2 step 3x777", "step", "gpt2", "bf16", 3, 777),
        # the benchmark's default workload
        _case("gpt2 step 8x1024", "step", "gpt2", "bf16", 8, 1024),
        # the micro-batch and the 24 layers that a GPU holds in the GPT-2 XL configuration, which has two pipeline stages
        # (width 1600, 25 heads: no multiple of a tile)
        _case("gpt2-xl step 4x1024", "step", "gpt2-xl", "bf16", 4, 1024, layers=24),
        # the LLaMA-3 1B configuration's batch on one GPU
        _case("llama3-1b step 4x2048", "step", "llama3-1b", "bf16", 4, 2048),
        # one layer of the 8B configuration: head dimension 128, grouped queries, long context
        _case("llama3-8b layer 1x4096", "layer", "llama3-8b", "bf16", 1, 4096),
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sampling", "evaluation", "prompt", "loop", "fp32", "step", "step", "large step", "layer"])
    if kind == "sampling":
        return _case(None, "logits", "gpt2", "bf16", rng.randint(1, 8), _between(rng, 16, 256))
    if kind == "evaluation":
        return _case(None, "logits", "gpt2", "bf16", rng.randint(1, 8), _between(rng, 256, 1024))
    if kind == "prompt":
        return _case(None, "logits", "llama3-1b", "bf16", rng.randint(1, 2), _between(rng, 64, 4096))
    if kind == "loop":
        return _case(None, "loop", "gpt2", "bf16", rng.randint(1, 8), _between(rng, 32, 1024), micro=rng.randint(1, 4),
                     clip=rng.choice([0.0, 1.0]))
    if kind == "fp32":
        return _case(None, "loop", "gpt2", "fp32", rng.randint(1, 4), _between(rng, 32, 512), micro=rng.randint(1, 2),
                     clip=rng.choice([0.0, 1.0]))
    if kind == "step":
        return _case(None, "step", "gpt2", "bf16", rng.randint(1, 8), _between(rng, 64, 1024))
    if kind == "large step":
        model, most = rng.choice([("gpt2-xl", 1024), ("llama3-1b", 2048)])
        return _case(None, "step", model, "bf16", rng.randint(1, 4), _between(rng, 128, most),
                     layers=24 if model == "gpt2-xl" else 0)
    return _case(None, "layer", "llama3-8b", "bf16", rng.randint(1, 2), _between(rng, 128, 4096))


# ------------------------------------------------------------------------------------------------- what is in hand
def _config(model, layers=0):
    cfg = (LLAMA3_PRESETS if model.startswith("llama3") else GPT2_PRESETS)[model]
    return dataclasses.replace(cfg, n_layer=layers or cfg.n_layer)


@functools.lru_cache(maxsize=None)
def _one_block(model, dtype):
    """The preset's modules with one block and a vocabulary of 128, whose tensors the real model's replace."""
    cfg = dataclasses.replace(_config(model), n_layer=1, vocab_size=128)
    if model.startswith("llama3"):
        return LLaMA3(cfg, device=DEVICE, dtype=dtype)
    return GPT2(dataclasses.replace(cfg, padded_vocab_size=128), device=DEVICE, dtype=dtype)


def _fill(module, cfg, gen):
    """GPT-2's and LLaMA-3's usual initial distributions, drawn on the GPU (the library's own initialisers draw on the
    host); biases and norms are moved off their constants, as training does."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() == 1:
                p.normal_(0.0 if name.endswith("bias") else 1.0, 0.02, generator=gen)
            elif name.endswith("c_proj.weight"):
                p.normal_(0.0, 0.02 / math.sqrt(2 * cfg.n_layer), generator=gen)
            else:
                # an embedding table of its own (LLaMA-3's) keeps nn.Embedding's unit normal, as the residual stream of a
                # trained model is larger than what one layer adds to it
                untied = name.endswith("wte.weight") and isinstance(module, LLaMA3)
                p.normal_(0.0, 1.0 if untied else 0.02, generator=gen)


def _model(case, gen):
    llama = case["model"].startswith("llama3")
    dtype = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    cfg = _config(case["model"], case["layers"])
    model = copy.deepcopy(_one_block(case["model"], dtype))
    model.config = cfg
    tr = model.transformer
    tr.add_module("h", tit.nn.Sequential(*[copy.deepcopy(tr["h"][0]) for _ in range(cfg.n_layer)]))
    rows = cfg.vocab_size if llama else cfg.padded_vocab_size
    tr["wte"].weight = torch.nn.Parameter(torch.empty(rows, cfg.n_embd, device=DEVICE, dtype=dtype))
    model.lm_head.weight = torch.nn.Parameter(torch.empty_like(tr["wte"].weight)) if llama else tr["wte"].weight
    _fill(model, cfg, gen)
    if not llama:
        with torch.no_grad():
            tr["wte"].weight[cfg.vocab_size:].zero_()
    return model, cfg


def _tokens(case, cfg, seed):
    gen = torch.Generator().manual_seed(seed)
    x = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), generator=gen)
    return x.pin_memory(), torch.roll(x, -1, dims=1).pin_memory()


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    do = case["do"]
    if do == "layer":
        cfg = _config(case["model"])
        block = copy.deepcopy(_one_block(case["model"], torch.bfloat16).transformer["h"][0])
        _fill(block, cfg, gen)
        shape = (case["batch"], case["seq"], cfg.n_embd)
        x = torch.randn(shape, device=DEVICE, generator=gen).bfloat16().requires_grad_()
        dy = torch.randn(shape, device=DEVICE, generator=gen).bfloat16()
        return {"do": do, "block": block, "flat": FlatParams(block.parameters()), "x": x, "dy": dy}
    model, cfg = _model(case, gen)
    if do == "logits":
        return {"do": do, "model": model, "x": _tokens(case, cfg, seed)[0]}
    opt = MixedPrecisionAdam(model.parameters(), lr=LEARNING_RATE, betas=(0.9, 0.95), weight_decay=0.1,
                             max_grad_norm=case["clip"])
    batches = [_tokens(case, cfg, seed * 16 + i) for i in range(case["micro"])]
    state = {"do": do, "model": model, "opt": opt, "batches": batches, "fused": case["dtype"] == "bf16"}
    if do == "step":
        step = TrainStep(model, opt, case["batch"], case["seq"], DEVICE, use_graph=True)
        step.idx.copy_(batches[0][0])
        step.tgt.copy_(batches[0][1])
        opt.set_lr(0.0)   # the eager steps before the capture leave the weights as they are
        step.prepare()
        opt.set_lr(LEARNING_RATE)
        state["step"] = step
    return state


# ------------------------------------------------------------------------------------------------- one pass
def run(state):
    do = state["do"]
    if do == "logits":
        with torch.no_grad():
            return state["model"](state["x"].to(DEVICE, non_blocking=True))
    if do == "layer":
        x = state["x"]
        x.grad = None
        state["flat"].mark_fresh()
        y = state["block"](x)
        y.backward(state["dy"])
        return {"y": y.detach(), "dx": x.grad, "grad": state["flat"].grad}
    opt = state["opt"]
    if do == "step":
        loss = state["step"](*state["batches"][0])
    else:
        opt.zero_grad()
        loss, micro = 0.0, len(state["batches"])
        for x, y in state["batches"]:
            x, y = x.to(DEVICE, non_blocking=True), y.to(DEVICE, non_blocking=True)
            _, part = state["model"](x, y, return_logits=not state["fused"])
            (part / micro).backward()
            loss += float(part.detach()) / micro
        opt.step()
    return {"loss": loss, "grad": opt.flat.grad, "param": opt.flat.param}


# ------------------------------------------------------------------------------------------------- what it needs
def work(case):
    cfg = _config(case["model"], case["layers"])
    llama = case["model"].startswith("llama3")
    C, tokens = cfg.n_embd, case["batch"] * case["seq"]
    if llama:
        hd = C // cfg.n_head
        qkv, ffn = (cfg.n_head + 2 * cfg.n_kv_head) * hd, 3 * C * cfg.ffn_dim
        head, tables = cfg.vocab_size * C, 2 * cfg.vocab_size * C
    else:
        qkv, ffn = 3 * C, 8 * C * C
        head = cfg.padded_vocab_size * C
        tables = head + cfg.block_size * C
    block = C * qkv + C * C + ffn
    elem = 4 if case["dtype"] == "fp32" else 2
    # causal attention: half of the T x T products, q k^T and p v
    attention = 2.0 * tokens * case["seq"] * C
    if case["do"] == "layer":
        # x, dy in, y, dx out, weights in, fp32 weight gradients out
        return {"bytes": tokens * C * 2 * 4 + block * (2 + 4), "flops": 6.0 * block * tokens + 3.5 * attention}
    dense = block * cfg.n_layer + head
    params = block * cfg.n_layer + tables
    if case["do"] == "logits":
        return {"bytes": params * elem + tokens * (8 + cfg.vocab_size * elem),
                "flops": 2.0 * dense * tokens + cfg.n_layer * attention}
    # the gradient is written, and read by the optimizer, which reads and writes two moments and the fp32 weights (and
    # writes the bf16 weights that the passes read)
    state = 4 + 4 + 8 + 8 + 8 + (2 + 2 if elem == 2 else 4)
    return {"bytes": params * state + tokens * 16 * case["micro"],
            "flops": case["micro"] * (6.0 * dense * tokens + 3.5 * cfg.n_layer * attention)}


def tolerance(case):
    # about four times what was measured against the same model in 64 bits, up to 3e-2 -- fp32 gradients: rel 4.5e-6, max
    # 2.5e-4; one layer: rel 5e-3, max 0.06; whole bf16 models, logits: rel 0.011; gradients: rel 0.010 (124M), 0.013 (XL,
    # 24 layers), 0.014 (LLaMA-3 1B), max 0.4 to 0.8 (the rms spans tensors of very different scale)
    if case["dtype"] == "fp32":
        return {"rel": 2e-5, "max": 2e-3}
    if case["do"] == "layer":
        return {"rel": 2e-2, "max": 0.25}
    return {"rel": 3e-2, "max": 0.99}

"""The work that a user of this framework has it do, as cases with sizes.

Six kinds of work, each through the entry points that a user's program calls:

* ``step``       one training step of a Llama-style decoder (``Trainer.train_step``: copy in, forward, recompute,
                 backward, gradient norm, AdamW, loss read back).  Widths are those of the configured models with
                 fewer layers and a smaller vocabulary, so that a state is made in about a second.
* ``eval``       the forward pass of a validation step (``GPTModel`` without gradients): hidden states and loss.
* ``linear``     forward, input gradient and accumulated weight gradient of one linear layer
                 (``kernels.gemm``), whole or as a tensor-parallel shard of it.
* ``attention``  causal grouped-query attention forward and backward on views of a packed QKV buffer
                 (``kernels.attention_fwd`` / ``attention_bwd``), plain or as a context-parallel rank's chunk.
* ``head``       vocabulary projection, cross entropy and their gradients (``OutputHead``).
* ``adamw``      gradient norm, clipping and update over flat buffers (``DistributedAdamW.step``).
"""
from __future__ import annotations

import math

import torch

from kareus_b200 import kernels as K
from kareus_b200.config import ModelConfig, ParallelConfig, TrainConfig, get_model_config
from kareus_b200.models.llama import OutputHead
from kareus_b200.parallel.collectives import CommFactory
from kareus_b200.train.optimizer import DistributedAdamW
from kareus_b200.train.trainer import Trainer, synthetic_batch

DEVICE = "cuda:0"
HEAD_DIM = 128
# configured models whose layer widths the cases use; `tiny128` is the smoke model and is small enough to be whole
WIDTHS = ("tiny128", "qwen3_1.7b", "llama3.2_3b", "llama3.1_8b")


def _step(name, model, layers, vocab, mbs, micro, seq, nano=2, recompute=True, kind="step"):
    return {"name": name, "kind": kind, "model": model, "layers": layers, "vocab": vocab, "mbs": mbs, "micro": micro,
            "seq": seq, "nano": nano, "recompute": recompute}


def _linear(name, tokens, n_in, n_out):
    return {"name": name, "kind": "linear", "tokens": tokens, "n_in": n_in, "n_out": n_out}


def _attention(name, sq, batch, groups, rep, q_offset=0):
    return {"name": name, "kind": "attention", "sq": sq, "batch": batch, "groups": groups, "rep": rep,
            "q_offset": q_offset}


def listed():
    return [
        # the smoke model as it is configured: launches and host work decide
        _step("step_smoke", "tiny128", 2, 2048, mbs=2, micro=2, seq=256),
        # the headline training run (3B width, micro batch 8 x 4096 tokens, recompute), two of its 28 layers
        _step("step_3b", "llama3.2_3b", 2, 16384, mbs=8, micro=1, seq=4096),
        # tied embeddings (1.7B width), two microbatches of a ragged sequence, activations kept instead of recomputed
        _step("step_1.7b", "qwen3_1.7b", 2, 32768, mbs=4, micro=2, seq=1900, recompute=False),
        # validation pass with per-head q/k norm over a sequence length that fits no tile, one nanobatch
        _step("eval_qknorm", "qwen3_1.7b", 2, 32768, mbs=3, micro=1, seq=2999, nano=1, kind="eval"),
        # gate/up projection of the 3B model for one nanobatch of the headline run
        _linear("linear_fc1", 16384, 3072, 16384),
        # QKV projection of the same model on one of eight tensor-parallel ranks: a narrow output
        _linear("linear_qkv_tp8", 16384, 3072, 640),
        # a short ragged batch through a small layer
        _linear("linear_small", 328, 1032, 776),
        # attention of one nanobatch of the headline run
        _attention("attn_4k", 4096, 4, 8, 3),
        # late chunk of a 16 k sequence on a context-parallel rank, heads of one of four tensor-parallel ranks
        _attention("attn_16k_chunk", 4096, 1, 2, 3, q_offset=12288),
        # short ragged sequences
        _attention("attn_short", 459, 2, 2, 2),
        # head and loss of the 3B model on a quarter of a nanobatch
        {"name": "head_128k", "kind": "head", "tokens": 4096, "hidden": 3072, "vocab": 128256},
        # optimizer over two layers' worth of 3B parameters
        {"name": "adamw_200m", "kind": "adamw", "matrices": 8, "rows": 8192, "cols": 3072},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "eval", "linear", "linear", "attention", "attention", "head", "adamw"))
    if kind in ("step", "eval"):
        model = rng.choice(WIDTHS)
        nano = rng.choice((1, 2))
        mbs = nano * rng.choice((1, 2, 3))
        cap = {"tiny128": 2048, "qwen3_1.7b": 4096, "llama3.2_3b": 3000, "llama3.1_8b": 2000}[model]
        vocab = {"tiny128": 2048}.get(model) or 128 * rng.randint(32, 160)
        c = _step("", model, 1 if model == "llama3.1_8b" else rng.choice((1, 2)), vocab, mbs, rng.choice((1, 2)),
                  _log_int(rng, 128, cap), nano, rng.choice((True, True, False)), kind)
    elif kind == "linear":
        # row strides of bf16 operands are multiples of 16 bytes, so feature counts are multiples of 8
        while True:  # no more work than the largest listed one
            c = _linear("", _log_int(rng, 64, 20000), 8 * _log_int(rng, 16, 1024), 8 * _log_int(rng, 16, 2048))
            if c["tokens"] * c["n_in"] * c["n_out"] <= 16384 * 3072 * 16384:
                break
    elif kind == "attention":
        while True:
            c = _attention("", _log_int(rng, 128, 16384), rng.choice((1, 2, 3, 4)), rng.choice((1, 2, 4, 8)),
                           rng.choice((1, 2, 3, 4)))
            if rng.random() < 0.3:
                c["q_offset"] = 128 * rng.randint(1, 96)
            if _pairs(c) * c["groups"] * c["rep"] * c["batch"] <= 4 * 24 * 4096 * 4096 // 2:
                break
    elif kind == "head":
        c = {"kind": "head", "tokens": _log_int(rng, 128, 4096), "hidden": rng.choice((2048, 3072, 4096)),
             "vocab": 8 * _log_int(rng, 500, 12000)}
    else:
        c = {"kind": "adamw", "matrices": rng.randint(1, 8), "rows": _log_int(rng, 64, 8192),
             "cols": rng.choice((512, 2048, 3072))}
    c.pop("name", None)
    return c


# ----------------------------------------------------------------------------- states
def _config(case) -> ModelConfig:
    cfg = get_model_config(case["model"]).replace(num_layers=case["layers"], vocab_size=case["vocab"],
                                                  max_seq_len=case["seq"])
    # The per-head q/k norm is part of the forward passes only: when these cases were chosen its backward on a GPU
    # gave a wrong key gradient, so a training step with it had no result to compare with.
    return cfg if case["kind"] == "eval" else cfg.replace(qk_layernorm=False)


def _trainer(case, seed, dtype="bf16") -> Trainer:
    tc = TrainConfig(micro_batch_size=case["mbs"], global_batch_size=case["mbs"] * case["micro"], seq_len=case["seq"],
                     seed=seed, dtype=dtype)
    par = ParallelConfig(num_nanobatches=case["nano"], recompute=case["recompute"])
    return Trainer(_config(case), par, tc, device=DEVICE)


def _randn(shape, gen, std=1.0, dtype=torch.bfloat16):
    t = torch.empty(shape, dtype=dtype, device=DEVICE)
    return t.normal_(0.0, std, generator=gen)


def prepare(case, seed):
    torch.cuda.set_device(DEVICE)
    kind = case["kind"]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    if kind in ("step", "eval"):
        trainer = _trainer(case, seed)
        batch = synthetic_batch(trainer.model_cfg, trainer.cfg, trainer.num_microbatches, seed=seed)
        if kind == "eval":
            trainer.model.eval()
        return {"kind": kind, "trainer": trainer, "batch": batch}
    if kind == "linear":
        n_in, n_out, t = case["n_in"], case["n_out"], case["tokens"]
        return {"kind": kind, "x": _randn((t, n_in), gen), "w": _randn((n_out, n_in), gen, 0.02),
                "dy": _randn((t, n_out), gen, 1e-3), "main_grad": _randn((n_out, n_in), gen, 1e-2, torch.float32)}
    if kind == "attention":
        sq, b, g, rep, d = case["sq"], case["batch"], case["groups"], case["rep"], HEAD_DIM
        packed = _randn((sq, b, g, (rep + 2) * d), gen)
        q = packed[..., : rep * d].unflatten(-1, (rep, d))
        if case["q_offset"]:
            # gathered keys of the whole sequence; this rank's queries start at q_offset
            kv = _randn((2, case["q_offset"] + sq, b, g, d), gen)
            k, v = kv[0], kv[1]
        else:
            k, v = packed[..., rep * d:(rep + 1) * d], packed[..., (rep + 1) * d:]
        return {"kind": kind, "q": q, "k": k, "v": v, "dout": _randn((sq, b, g * rep, d), gen, 1e-3),
                "q_offset": case["q_offset"], "scale": 1.0 / math.sqrt(d)}
    if kind == "head":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        cfg = get_model_config("llama3.2_3b").replace(hidden_size=h, vocab_size=v)
        weight = torch.nn.Parameter(_randn((v, h), gen, 0.02))
        weight.main_grad = torch.zeros(v, h, dtype=torch.float32, device=DEVICE)
        head = OutputHead(cfg, ParallelConfig(), CommFactory(), torch.bfloat16, DEVICE, 0, tied_weight=weight)
        return {"kind": kind, "head": head, "x": _randn((t, 1, h), gen),
                "labels": torch.randint(0, v, (t, 1), device=DEVICE, generator=gen),
                "loss_weight": torch.full((t, 1), 1.0 / t, device=DEVICE)}
    if kind == "adamw":
        params = [torch.nn.Parameter(_randn((case["rows"], case["cols"]), gen, 0.02)) for _ in range(case["matrices"])]
        opt = DistributedAdamW(params, TrainConfig())
        opt.grad_flat.normal_(0.0, 1e-3, generator=gen)
        return {"kind": kind, "opt": opt}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "step":
        tr = state["trainer"]
        loss = tr.train_step(state["batch"])
        return {"loss": loss, "grads": tr.optimizer.grad_flat, "weights": tr.optimizer.param_flat,
                "master": tr.optimizer.master}
    if kind == "eval":
        tr = state["trainer"]
        model, batch = tr.model, tr.to_device(state["batch"])
        with torch.no_grad():
            hidden = model.run_block(model.embed(batch["tokens"]))
            loss = model.head_loss(hidden, batch["labels"], batch["loss_mask"],
                                   loss_denominator=float(batch["tokens"].numel()))
        return {"hidden": hidden, "loss": loss}
    if kind == "linear":
        x, w, dy = state["x"], state["w"], state["dy"]
        y = K.gemm(x, w, trans_b=True)
        dx = K.gemm(dy, w, trans_b=False)
        dw = K.gemm(dy, x, trans_a=True, trans_b=False, accumulate=state["main_grad"])
        return {"y": y, "dx": dx, "dw": dw}
    if kind == "attention":
        q, k, v, scale, off = state["q"], state["k"], state["v"], state["scale"], state["q_offset"]
        out, lse = K.attention_fwd(q, k, v, scale, causal=True, q_offset=off)
        dq, dk, dv = K.attention_bwd(state["dout"], q, k, v, out, lse, scale, causal=True, q_offset=off)
        return {"out": out, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    if kind == "head":
        head, x = state["head"], state["x"].detach().requires_grad_()
        loss = head(x, state["labels"], state["loss_weight"])
        loss.backward()
        return {"loss": loss.detach(), "dx": x.grad, "dw": head.weight.main_grad}
    opt = state["opt"]
    norm = opt.step()
    return {"norm": norm, "weights": opt.param_flat, "master": opt.master, "exp_avg": opt.m, "exp_avg_sq": opt.v}


# ----------------------------------------------------------------------------- work and tolerance
def _pairs(case) -> float:
    """Visible (query, key) pairs of one head: query i sees keys 0 .. q_offset + i."""
    sq = case["sq"]
    return sq * case["q_offset"] + sq * (sq + 1) / 2


def work(case):
    kind = case["kind"]
    if kind in ("step", "eval"):
        cfg = _config(case)
        tokens = case["mbs"] * case["micro"] * case["seq"]
        n = cfg.num_params()
        if kind == "eval":
            h, v = cfg.hidden_size, cfg.vocab_size
            layer = cfg.flops_per_token(case["seq"], recompute=False) - 6.0 * h * v
            return {"bytes": 2.0 * n + 20.0 * tokens, "flops": tokens * (layer / 3.0 + 2.0 * h * v)}
        # weights read; fp32 gradient written and read; fp32 master, m, v read and written; bf16 weight written
        return {"bytes": 36.0 * n + 20.0 * tokens,
                "flops": tokens * cfg.flops_per_token(case["seq"], recompute=case["recompute"])}
    if kind == "linear":
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        return {"bytes": 2.0 * (2 * t * i + 2 * t * o + o * i) + 8.0 * o * i, "flops": 6.0 * t * i * o}
    if kind == "attention":
        sq, b, g, hq = case["sq"], case["batch"], case["groups"], case["groups"] * case["rep"]
        skv = sq + case["q_offset"]
        q_like, kv_like = sq * b * hq * HEAD_DIM * 2.0, skv * b * g * HEAD_DIM * 2.0
        return {"bytes": 4 * q_like + 4 * kv_like + 4.0 * b * hq * sq,
                "flops": 14.0 * _pairs(case) * HEAD_DIM * b * hq}
    if kind == "head":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        return {"bytes": 4.0 * t * h + 10.0 * v * h + 16.0 * t, "flops": 6.0 * t * h * v}
    n = case["matrices"] * case["rows"] * case["cols"]
    return {"bytes": 30.0 * n, "flops": 15.0 * n}


def tolerance(case):
    # About four times the distance of one pass from the same statements in 64 bits.  A training step at 3B width is
    # 1.4e-2 (rel) and 0.3 (max) away from them in its gradients, since every activation is rounded to bf16; attention
    # 3e-3 and 0.08 (P and dS are rounded to bf16), hidden states 1e-2 and 0.06, other matrix products 1.7e-3 and
    # 4e-3 (rounding of the result), the optimizer's bf16 weights 2e-5 and one unit in the last place.
    return {
        "step": {"rel": 3e-2, "max": 0.95},
        "eval": {"rel": 3e-2, "max": 0.25},
        "linear": {"rel": 7e-3, "max": 1.6e-2},
        "attention": {"rel": 1.2e-2, "max": 0.33},
        "head": {"rel": 7e-3, "max": 2e-2},
        "adamw": {"rel": 1e-4, "max": 1e-2},
    }[case["kind"]]

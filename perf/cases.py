"""The measured workloads: training steps and scoring passes through the public ``Trainer``.

A training case is one optimizer step as the trainers of ``surogate pt`` / ``surogate sft`` take it: host token arrays in, loss and
gradient norm back on the host, weights and optimizer state updated.  A scoring case is ``Trainer.token_logprobs`` over a batch, the
pass that DPO and GRPO make for their reference log-probabilities.  Widths (hidden sizes, head counts, MLP widths, vocabulary,
expert counts), sequence lengths, micro-batches, recipes and optimizers are those of ``bench.py``, ``examples/`` and ``tests/``; the
layer stacks are cut to a few layers so that several independent trainers fit one GPU.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from surogate_b200.runtime.trainer import Trainer, TrainerConfig

VOCAB = 151936

# hidden size, query heads, KV heads, MLP width, tied embeddings (head size 128 throughout)
WIDTHS = {
    "d512": (512, 4, 2, 1536, True),
    "d1024": (1024, 16, 8, 3072, True),
    "d2048": (2048, 16, 8, 6144, True),
    "d4096": (4096, 32, 8, 12288, False),
    "d5120": (5120, 40, 8, 17408, False),
    "moe2048": (2048, 32, 4, 768, False),   # MLP width of one expert
}

BASE = dict(mode="train", width="d1024", layers=2, vocab=VOCAB, batch=1, seq=1024, accum=1, recipe="bf16", optimizer="adamw_8bit", recompute=False,
            graphs=False, lora_rank=0, qlora="", packed=False, masked=0.0, drop_ignored=False, experts=0, top_k=0)


def case(name=None, **kw):
    c = dict(BASE, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One short sequence scored on a small model: a handful of kernels per layer, so launches and host work are the whole cost.
        case("score_small", mode="score", width="d512", layers=2, vocab=4096, batch=1, seq=128),
        # The smallest training run of the benchmark (smoke tests, debugging runs, the first minutes of every new configuration).
        case("train_small", width="d512", layers=2, vocab=4096, batch=2, seq=512),
        # Full fine-tune of a 0.6B-wide model as `surogate sft` runs it by default: bf16, CUDA-graph replay, fp32 AdamW moments.
        case("train_d1024_bf16_graphs", width="d1024", layers=6, batch=8, seq=2048, optimizer="adamw", graphs=True),
        # A sequence length that is no multiple of a tile (a cut-to-fit instruction dataset), with activation recompute.
        case("train_d1024_ragged", width="d1024", layers=4, batch=3, seq=1000, recompute=True),
        # Pre-training with NorMuon on the hidden matrices.
        case("train_d1024_normuon", width="d1024", layers=4, batch=4, seq=2048, optimizer="normuon"),
        # The headline pre-training configuration: 8B width, FP8-hybrid, 8-bit AdamW, sequence 4096, micro-batch 2.
        case("train_d4096_fp8", width="d4096", layers=4, batch=2, seq=4096, recipe="fp8_hybrid"),
        # The same width under the NVFP4 recipe.
        case("train_d4096_nvfp4", width="d4096", layers=3, batch=2, seq=2048, recipe="nvfp4"),
        # The other headline model: mixture of 128 experts, 8 per token, NVFP4 dense projections and FP8 experts.
        case("train_moe_nvfp4", width="moe2048", layers=2, batch=1, seq=4096, recipe="nvfp4", experts=128, top_k=8),
        # Supervised LoRA fine-tuning of a 14B width on long rows, no loss on the prompt quarter of each row.
        case("lora_d5120_long", width="d5120", layers=2, batch=1, seq=8192, lora_rank=16, masked=0.25, recompute=True),
        # LoRA under FP8-hybrid on packed documents with gradient accumulation; prompt rows stay out of the vocabulary GEMMs.
        case("lora_d4096_packed_fp8", width="d4096", layers=3, batch=2, seq=2048, accum=2, recipe="fp8_hybrid", lora_rank=16, packed=True, masked=0.5,
             drop_ignored=True),
        # QLoRA: the frozen base stored as NF4 blocks and rebuilt layer by layer.
        case("qlora_d5120_nf4", width="d5120", layers=2, batch=2, seq=2048, lora_rank=16, qlora="bnb_nf4", recompute=True),
        # Reference log-probabilities of preference pairs, rows padded to their longest member.
        case("score_d4096", mode="score", width="d4096", layers=4, batch=4, seq=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["score", "bf16", "bf16", "fp8", "nvfp4", "moe", "lora", "lora_fp8", "qlora"])
    kw = {}
    if kind == "score":
        kw.update(mode="score", width=rng.choice(["d512", "d1024", "d2048", "d4096"]))
    elif kind == "bf16":
        kw.update(width=rng.choice(["d512", "d1024", "d2048", "d4096"]), optimizer=rng.choice(["adamw_8bit", "adamw", "adamw_8bit", "normuon"]),
                  recompute=rng.random() < 0.5, graphs=rng.random() < 0.4)
    elif kind == "fp8":
        kw.update(width=rng.choice(["d1024", "d2048", "d4096"]), recipe="fp8_hybrid", graphs=rng.random() < 0.4)
    elif kind == "nvfp4":
        kw.update(width=rng.choice(["d1024", "d2048", "d4096"]), recipe="nvfp4")
    elif kind == "moe":
        kw.update(width="moe2048", recipe=rng.choice(["bf16", "fp8_hybrid", "nvfp4"]), experts=rng.choice([8, 32, 64, 128]), top_k=rng.choice([2, 4, 8]))
    else:
        kw.update(width=rng.choice(["d1024", "d4096", "d5120"]), lora_rank=rng.choice([8, 16, 32]), recompute=rng.random() < 0.5,
                  recipe="fp8_hybrid" if kind == "lora_fp8" else "bf16", qlora="bnb_nf4" if kind == "qlora" else "",
                  masked=rng.choice([0.0, 0.25, 0.5]), drop_ignored=rng.random() < 0.3)
    small = kw["width"] == "d512"
    kw["vocab"] = 4096 if small else VOCAB
    kw["layers"] = rng.randint(1, 2 if kind == "moe" else 3)
    # tokens of one pass, then a sequence length that divides them: tile multiples, packed rows and odd lengths
    tokens = _log_int(rng, 128, 8192)
    shape = rng.choice(["tile", "packed", "odd"]) if kind != "score" else rng.choice(["tile", "odd"])
    seq = min(tokens, _log_int(rng, 96, 4096))
    if shape != "odd":
        seq = max(128, seq // 128 * 128)
    else:
        seq = min(seq, 2048) | 1
    kw["seq"] = seq
    kw["batch"] = max(1, min(8, tokens // seq))
    kw["packed"] = shape == "packed"
    if shape == "packed":
        kw["graphs"] = False
    if kw.get("mode") != "score" and kind != "moe" and kw["batch"] >= 2 and rng.random() < 0.25:
        kw["accum"], kw["batch"] = 2, kw["batch"] // 2
    return case(**kw)


# ------------------------------------------------------------------------------------------------ what a pass needs
def _params(c):
    """(parameters of all weight matrices, those a token goes through, parameters of the embedding table) without norms."""
    d, hq, hkv, ff, tied = WIDTHS[c["width"]]
    att = d * (hq + 2 * hkv) * 128 + hq * 128 * d
    if c["experts"]:
        mlp, mlp_active = c["experts"] * 3 * d * ff + c["experts"] * d, c["top_k"] * 3 * d * ff + c["experts"] * d
    else:
        mlp = mlp_active = 3 * d * ff
    head = c["vocab"] * d
    return c["layers"] * (att + mlp) + head, c["layers"] * (att + mlp_active) + head, 0 if tied else head


def work(c):
    d, hq, hkv, ff, _ = WIDTHS[c["width"]]
    n_all, n_active, n_emb = _params(c)
    tokens = c["accum"] * c["batch"] * c["seq"]
    att = c["layers"] * c["accum"] * c["batch"] * 2.0 * c["seq"] * c["seq"] * hq * 128     # causal Q.K^T and P.V
    if c["packed"]:
        att /= 4
    if c["mode"] == "score":
        return {"bytes": 2.0 * n_all + 12 * tokens, "flops": 2.0 * n_active * tokens + att}
    head = c["vocab"] * d
    loss_tokens = tokens * (1 - c["masked"]) if c["drop_ignored"] else tokens
    if c["lora_rank"]:
        # forward and input gradients of the frozen base; adapters are small beside it
        flops = 4.0 * (n_active - head) * tokens + 4.0 * head * loss_tokens + 3.5 * att
        base = (n_all - head) * (0.53 if c["qlora"] else 2.0) + 2.0 * head
        return {"bytes": base + 8 * tokens, "flops": flops}
    flops = 6.0 * (n_active - head) * tokens + 6.0 * head * loss_tokens + 3.5 * att
    state = {"adamw_8bit": 2.125, "adamw": 8.0, "normuon": 2.125}[c["optimizer"]]
    return {"bytes": (n_all + n_emb) * (2 + 2 + 2 + 2 * state) + 8 * tokens, "flops": flops}


# ------------------------------------------------------------------------------------------------ state of a user's program
def _model(c):
    d, hq, hkv, ff, tied = WIDTHS[c["width"]]
    m = dict(vocab_size=c["vocab"], d_model=d, n_layers=c["layers"], num_query_heads=hq, num_kv_heads=hkv, head_size=128, tie_word_embeddings=tied)
    if c["experts"]:
        return dict(m, architecture="Qwen3MoeForCausalLM", moe_d_ff=ff, num_experts=c["experts"], num_experts_per_tok=c["top_k"], aux_loss_coef=1e-3)
    return dict(m, architecture="Qwen3ForCausalLM", d_ff=ff)


def _load_weights(tr, seed):
    """A checkpoint's worth of weights, made on the GPU: N(0, 0.02) matrices, norm weights around one."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for p in tr.cm.params:
        if p.tied_to:
            continue
        t = torch.randn(tuple(p.spec.shape), generator=gen, device="cuda", dtype=torch.float32)
        tr.store.load_tensor(p.name, t.mul_(0.05).add_(1.0) if p.spec.init == "ones" else t.mul_(0.02))
    tr.store.sync_work_from_master()
    tr.recipe.on_weights_updated(tr.store)


def _batch(c, seed):
    """Token ids with the skew of natural text (a few frequent ones, a long tail), targets = next token, ignored on the prompt part."""
    rng = np.random.default_rng(seed)
    rows, T = c["accum"] * c["batch"], c["seq"]
    ids = (c["vocab"] * rng.random((rows, T + 1)) ** 3).astype(np.int32)
    x, y = ids[:, :-1].copy(), ids[:, 1:].copy()
    pos = None
    starts = [[0] for _ in range(rows)]
    if c["packed"]:
        pos = np.empty((rows, T), dtype=np.int32)
        for r in range(rows):
            cuts = sorted(set(int(v) for v in rng.integers(1, T, size=min(5, T - 1))) | {0, T})
            starts[r] = cuts[:-1]
            for a, b in zip(cuts[:-1], cuts[1:]):
                pos[r, a:b] = np.arange(b - a, dtype=np.int32)
                y[r, b - 1] = -100                                   # the last token of a document predicts nothing
    if c["masked"]:
        for r in range(rows):
            ends = starts[r][1:] + [T]
            for a, b in zip(starts[r], ends):
                y[r, a:a + int((b - a) * c["masked"])] = -100        # prompt part
    return x, y, pos


def prepare(c, seed):
    lora = None
    if c["lora_rank"]:
        lora = dict(rank=c["lora_rank"], alpha=2 * c["lora_rank"], dropout=0.0, dtype="fp32", rslora=False, train_router=False,
                    targets=["q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj"])
    cfg = TrainerConfig(model=_model(c), batch_size=c["batch"], seq_len=c["seq"], grad_accum=c["accum"], recipe=c["recipe"], optimizer=c["optimizer"],
                        learning_rate=2e-4 if lora else 3e-4 if c["optimizer"] == "normuon" else 1e-5, weight_decay=0.1, recompute=c["recompute"], use_cuda_graphs=c["graphs"], lora=lora, qlora=c["qlora"] or None,
                        lmhead_drop_ignored_rows=c["drop_ignored"])
    tr = Trainer(cfg, device=torch.device("cuda", torch.cuda.current_device()))
    if c["qlora"]:
        tr.init_weights(seed)                     # quantises the frozen base as it is laid out
    else:
        _load_weights(tr, seed)
    if tr.lora is not None:
        if not c["qlora"]:
            tr.lora.init_weights(seed)
        # an adapter that has been trained for a while: its B matrices are no longer zero
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        tr.lora.master.add_(torch.randn(tr.lora.master.shape, generator=gen, device="cuda"), alpha=2e-3)
        tr.lora.sync_work()
    state = {"trainer": tr, "case": c, "batch": _batch(c, seed)}
    if c["mode"] == "train":
        # a run in progress: scaling histories, optimizer moments and captured graphs exist
        for _ in range(3 if c["graphs"] else 2):
            x, y, pos = state["batch"]
            tr.step(x, y, pos)
    return state


def run(state):
    tr, c = state["trainer"], state["case"]
    x, y, pos = state["batch"]
    if c["mode"] == "score":
        return tr.token_logprobs(x, y, pos)
    out = tr.step(x, y, pos)
    r = {"loss": out["loss"]}
    bf16 = c["recipe"] == "bf16"
    if tr.lora is not None:
        r["adapters"] = tr.lora.master
        if bf16:                                  # the moments are exponential averages of the adapters' gradients
            r["m"], r["v"] = tr.lora.opt_state["m"], tr.lora.opt_state["v"]
        return r
    r["weights"] = {name: b.master for name, b in tr.store.buckets.items()}
    if bf16 and not c["experts"] and c["optimizer"] != "normuon":
        r["grads"] = {name: b.grad for name, b in tr.store.buckets.items() if b.layer is not None}
    return r


def tolerance(c):
    """Limits at about four times the distance between the kernels and the same steps on PyTorch library ops (``backend="ref"``), as
    measured at the listed sizes on a B200."""
    if c["mode"] == "score":
        return {"rel": 5e-3, "max": 0.02}         # measured 1.2e-3 and 4.9e-3: bf16 logits of a few layers
    if c["lora_rank"]:
        return {"rel": 0.03, "max": 0.9}          # bf16: 8.9e-3 and 0.22, set by the second moments; FP8 steps return the adapters alone
    if c["recipe"] == "fp8_hybrid":
        return {"rel": 0.01, "max": 0.1}          # weights 3.6e-4 and 1.2e-2, the loss of short batches moves more
    if c["recipe"] == "nvfp4":
        return {"rel": 0.02, "max": 0.1}          # weights 6.4e-4 and 1.8e-2, loss 9.3e-3: stochastic rounding of 4-bit gradients
    if c["experts"] or c["optimizer"] == "normuon":
        return {"rel": 0.01, "max": 0.3}          # weights only: 9.3e-4 and 7.6e-2 after three orthogonalised updates
    return {"rel": 0.03, "max": 0.6}              # gradients of the blocks: 1.3e-2 and 0.15 after a bf16 backward pass

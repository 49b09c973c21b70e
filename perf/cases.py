"""The work that a user of this framework has it do: whole training steps (``fwd_bwd`` + ``step``) and held-out
evaluation through the public API, on slices in depth of the packaged models.  A layer costs the same at every depth,
so a few layers stand for the whole model; width, vocabulary, sequence lengths and options are the real ones.

``listed()`` are the measured cases, ``draw(rng)`` gives further ones of the same ranges.  A case names a packaged model
(or the hybrid of this file), the layers taken of it, the tokens of one step, how they fall into sequences, and the
options in use:

* ``task``     ``full`` (every weight trained), ``lora`` (rank-r adapters on every projection), ``eval`` (loss only)
* ``tokens``   in one step, as sequences of ``shortest`` to ``longest`` tokens (equal: all that long, a last one shorter)
* ``masked``   supervised fine-tuning: the first part of every sequence, the prompt, carries no loss
* ``optimizer``  ``adamw`` (fp32 state), ``adamw16`` (bf16 state), ``muon`` (matrices by Muon, the rest by AdamW)
* ``clip``     clip the gradient's global norm before the update
"""
import json
import math
import os
import random
import zlib

import torch

import flextrain_b200 as ft
from flextrain_b200.io.sequence import Sequence

GIB = 1 << 30

with open(os.path.join(os.path.dirname(ft.__file__), "configs", "model_dims.json")) as _f:
    MODELS = json.load(_f)

# Gated-DeltaNet hybrid with a dense feed-forward: the mixers of the packaged 80B hybrid at its width, three linear
# layers to one of full attention.
MODELS["hybrid_dense"] = dict(
    MODELS["qwen3_next_80B_A3B"], arch="qwen3_5", expert_dim=6144, num_routed_experts=0, top_k=0, num_shared_experts=0,
    shared_dim=0)


def _case(name, model, layers, tokens, shortest, longest, task="full", optimizer="adamw", masked=False, clip=False):
    return {"name": name, "model": model, "layers": layers, "tokens": tokens, "shortest": shortest, "longest": longest,
            "task": task, "optimizer": optimizer, "masked": masked, "clip": clip}


def listed():
    return [
        # the smallest call: the packaged quick-start run, where launches and host time count
        _case("quickstart_tiny", "tiny_llama", 2, 512, 128, 128),
        # a small adapter run on short chat turns, ragged, as the packaged fine-tuning example has them
        _case("lora_short_chat", "llama3_2_1B", 6, 3001, 20, 512, task="lora", masked=True),
        # small-model pretraining, speed-run style: Muon for the matrices
        _case("pretrain_muon", "nanogpt_124M", 6, 16384, 1024, 1024, optimizer="muon"),
        # the headline: full fine-tuning at sequence length 1024
        _case("full_8b", "llama3_1_8B", 6, 16384, 1024, 1024),
        # adapters on every projection of the same model over packed instruction data
        _case("lora_8b_sft", "llama3_1_8B", 6, 16384, 64, 2048, task="lora", masked=True),
        # full fine-tuning of a small model with per-head norms and a tied head on ragged data, clipped
        _case("sft_ragged", "qwen3_0_6B", 6, 9377, 17, 2048, masked=True, clip=True),
        # routed experts, few and wide: pretraining batches
        _case("moe_64", "olmoe_1B_7B", 4, 16384, 2048, 2048),
        # routed experts, many and narrow, a smaller ragged batch, bf16 state
        _case("moe_128_sft", "qwen3_30B_A3B", 3, 8000, 64, 2048, optimizer="adamw16", masked=True),
        # Gated DeltaNet layers with gated attention
        _case("hybrid_linear", "hybrid_dense", 4, 16384, 512, 4096),
        # sandwich norms, sliding windows, 256-wide heads, a large vocabulary
        _case("gemma_sliding", "gemma3_1B", 6, 8192, 256, 4096),
        # one long sequence, worked through in chunks over a window of keys
        _case("long_context", "dense_12B_long", 4, 32768, 32768, 32768),
        # loss on held-out data: forward only
        _case("evaluate_8b", "qwen3_8B", 6, 12000, 33, 4096, task="eval"),
    ]


# What draw() may take: (model, most layers, fewest and most tokens, longest sequence, tasks, optimizers)
_RANGES = [
    ("tiny_llama", 2, 64, 4096, 512, ("full", "lora", "eval"), ("adamw", "adamw16", "muon")),
    ("llama3_2_1B", 6, 512, 16384, 2048, ("full", "lora", "eval"), ("adamw", "adamw16")),
    ("nanogpt_124M", 6, 1024, 32768, 2048, ("full", "eval"), ("adamw", "muon")),
    ("llama3_1_8B", 5, 1024, 16384, 4096, ("full", "lora", "eval"), ("adamw", "adamw16")),
    ("qwen3_0_6B", 6, 512, 16384, 4096, ("full", "lora", "eval"), ("adamw", "adamw16", "muon")),
    ("qwen3_8B", 5, 1024, 16384, 4096, ("full", "lora", "eval"), ("adamw", "adamw16")),
    ("olmoe_1B_7B", 4, 1024, 16384, 4096, ("full", "eval"), ("adamw", "adamw16")),
    ("qwen3_30B_A3B", 3, 1024, 16384, 4096, ("full", "eval"), ("adamw16",)),
    ("hybrid_dense", 4, 512, 16384, 8192, ("full", "eval"), ("adamw", "adamw16")),
    ("gemma3_1B", 6, 512, 8192, 4096, ("full", "eval"), ("adamw", "adamw16")),
    ("dense_12B_long", 3, 16384, 32768, 32768, ("full", "eval"), ("adamw", "adamw16")),
]


def draw(rng):
    model, most, lo, hi, longest, tasks, optimizers = rng.choice(_RANGES)
    tokens = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    task = rng.choice(tasks)
    layers = 4 if model == "hybrid_dense" else 6 if model == "gemma3_1B" else rng.randint(1 if most < 4 else 2, most)
    if model == "dense_12B_long":
        top = low = tokens                        # this one is for single long sequences
    else:
        top = min(tokens, int(round(math.exp(rng.uniform(math.log(32), math.log(longest))))))
        top = max(top, tokens // 512)             # a step holds some hundred sequences at most
        low = top if rng.random() < 0.3 else max(2, top // rng.choice((4, 16, 64)))
    return {"model": model, "layers": layers, "tokens": tokens, "shortest": low, "longest": top, "task": task,
            "optimizer": "adamw" if task == "eval" else rng.choice(optimizers),
            "masked": task != "eval" and rng.random() < 0.5, "clip": task == "full" and rng.random() < 0.3}


def _lengths(case):
    """The sequence lengths of a case: even in their logarithm, and the same for every seed."""
    plain = {k: v for k, v in case.items() if k != "name"}
    rng = random.Random(zlib.crc32(json.dumps(plain, sort_keys=True).encode()))
    lo, hi, left, out = case["shortest"], case["longest"], case["tokens"], []
    while left > 0:
        n = min(left, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))
        if left - n == 1:                         # no sequence of a single token
            n = n + 1 if n < hi else n - 1
        out.append(n)
        left -= n
    return out


def _dims(case):
    d = {k: v for k, v in MODELS[case["model"]].items() if k not in ("arch", "hyperparams")}
    moe = bool(d.get("num_routed_experts"))
    d.update(n_layers=case["layers"], ffn_dim=d["expert_dim"], num_routed_experts=d.get("num_routed_experts", 0),
             top_k=d.get("top_k", 0), num_shared_experts=d.get("num_shared_experts", 0) if moe else 0, is_causal=True)
    return d


def _optimizer(case):
    if case["optimizer"] == "muon":
        return ft.HybridMuonAdamW(muon=ft.Muon(lr=1e-3), adamw=ft.AdamW(lr=3e-4, state_dtype=torch.float32))
    state = torch.float32 if case["optimizer"] == "adamw" else torch.bfloat16
    return ft.AdamW(lr=1e-4, beta1=0.9, beta2=0.95, weight_decay=0.01, state_dtype=state)


def _sequences(case, vocab, seed):
    g = torch.Generator().manual_seed(seed)
    out = []
    for i, n in enumerate(_lengths(case)):
        ids = torch.randint(0, vocab, (n,), generator=g)
        mask = None
        if case["masked"]:
            mask = torch.ones(n)
            mask[: n // 3] = 0
        out.append(Sequence(ids.pin_memory(), targets=torch.roll(ids, -1).pin_memory(), loss_mask=mask, seq_id=i))
    return out


def _runs(tensors):
    """Neighbouring matrices in an arena as one flat view each, so that a step's results are few tensors."""
    groups = []
    for t in tensors:
        if t.dtype == torch.float32:              # norm gains and the like, see _vectors: a run ends there
            groups.append([])
        elif groups and groups[-1]:
            groups[-1].append(t)
        else:
            groups.append([t])
    out = []
    for g in filter(None, groups):
        first, last = g[0].view(-1), g[-1].view(-1)
        n = last.storage_offset() + last.numel() - first.storage_offset()
        out.append(torch.as_strided(first, (n,), (1,)))
    return out


def _vectors(tensors):
    """The small fp32 tensors (norm gains, gate parameters)."""
    return [t.view(-1) for t in tensors if t.dtype == torch.float32]


def _condition(am, seed):
    """Random weights with the balance of a trained model.  The embedding sets the residual stream and each branch adds a
    little to it (small residual projections, as depth-scaled initialisation has them), and the routers decide clearly
    and share the load: the stream of every token holds the directions of its ``top_k`` experts in every layer."""
    tied, routers = am.head.tied, []
    for _, _, name, t in am.named_master_params():
        if name == "w_tok_embeddings":
            table = t.mul_(2.0 if tied else 50.0)
        elif name in ("w_o", "w_2", "w_down", "w_lin_out"):
            t.mul_(1 / 64 if tied else 1 / 16)
        elif name in ("w_post_attn_norm", "w_post_ffn_norm"):
            t.mul_(0.25)
        elif name == "w_router":
            routers.append(t)
    if routers:
        g = torch.Generator(device=table.device).manual_seed(seed + 1)
        top_k = am.model_config.top_k
        for r in routers:
            ways = torch.nn.functional.normalize(r.float(), dim=1)
            mine = torch.rand(table.shape[0], r.shape[0], generator=g, device=r.device).topk(top_k, dim=1).indices
            table.add_((8.0 * ways[mine].sum(1)).to(table.dtype))
    if tied:
        am.buffers.head_params()["w_head_proj"].copy_(am.buffers.embed_params()["w_tok_embeddings"])


class State:
    """What a training program holds: the model, the data of the step, and where its results are."""


def prepare(case, seed):
    dims = _dims(case)
    model = MODELS[case["model"]]
    s = State()
    s.case = case
    lora = dict(lora_targets="all", lora_rank=16, lora_alpha=16.0) if case["task"] == "lora" else {}
    s.am = ft.from_dims(dims, arch=model["arch"], optimizer=_optimizer(case), max_seq_len=case["longest"],
                        max_global_batch_tokens=case["tokens"], max_gpu_mem_bytes=48 * GIB,
                        max_host_mem_bytes=32 * GIB, device="cuda:0", hyperparams=model["hyperparams"],
                        init_seed=seed, init_on_device=True, **lora)
    _condition(s.am, seed)
    s.seqs = _sequences(case, dims["vocab_size"], seed)
    s.results, s.vectors = {}, {}
    if case["task"] == "eval":
        return s
    if case["task"] == "lora":                    # the adapters start away from zero, as they are after a few steps
        g = torch.Generator(device="cuda:0").manual_seed(seed)
        for _, _, name, t in s.am.named_master_params():
            if name.endswith("_lora_b"):
                t.normal_(0.0, 0.003, generator=g)
    am, bm, layers = s.am, s.am.buffers, range(case["layers"])
    keep = lambda spec, p: [p[t.name] for t in spec.trainable()]
    grads = [list(bm.grads(l).values()) for l in layers] + [list(bm.embed_grads().values()), list(bm.head_grads().values())]
    weights = [keep(am.layers[l].param_spec, bm.params(l)) for l in layers] + [
        keep(am.embed.param_spec, bm.embed_params()), keep(am.head.param_spec, bm.head_params())]
    for name, units in (("grads", grads), ("weights", weights)):
        s.results[name] = [_runs(u) for u in units]
        s.vectors[name] = [v for u in units for v in _vectors(u)]
    return s


def run(s):
    if s.case["task"] == "eval":
        stats = s.am.evaluate(s.seqs)
        return {"loss": stats.loss, "token_losses": torch.cat([q.per_token_loss for q in s.seqs])}
    stats = s.am.fwd_bwd(s.seqs)
    s.am.step(max_grad_norm=1.0 if s.case["clip"] else None)
    return {"loss": stats.loss, **s.results, **{k + "_1d": torch.cat(v) for k, v in s.vectors.items() if v}}


def work(case):
    d, hyper = _dims(case), MODELS[case["model"]]["hyperparams"]
    T, L, dm, hd = case["tokens"], case["layers"], d["d_model"], d["head_dim"]
    lens = _lengths(case)
    q, kv = d["n_heads"] * hd, d["n_kv_heads"] * hd
    gated = MODELS[case["model"]]["arch"].startswith("qwen3_5")
    window = hyper.get("sliding_window", 0)
    pattern = hyper.get("layer_pattern", "")
    kinds = "LLLF" if pattern == "3L1F" else "SSSSSF" if pattern == "5S1F" else "F"
    kinds = [kinds[i % len(kinds)] for i in range(L)]
    experts, k = d["num_routed_experts"], d["top_k"]
    seen = lambda w: float(sum(n * (n + 1) // 2 if not w or n <= w else w * (w + 1) // 2 + (n - w) * w for n in lens))
    weights = active = core = 0.0
    for kind in kinds:
        if kind == "L":
            g = hyper["gdn"]
            key, val = g["n_k_heads"] * g["head_k_dim"], g["n_v_heads"] * g["head_v_dim"]
            mix = dm * (2 * key + 2 * val + 2 * g["n_v_heads"]) + val * dm
            core += 4 * 2.0 * T * g["n_v_heads"] * g["head_k_dim"] * g["head_v_dim"]
        else:
            mix = dm * (q * (2 if gated else 1) + 2 * kv) + q * dm
            core += 4.0 * seen(window if kind == "S" else 0) * q
        ffn = 3 * dm * d["expert_dim"]
        weights += mix + (experts * ffn + dm * experts if experts else ffn)
        active += mix + (k * ffn + dm * experts if experts else ffn)
    head = float(d["vocab_size"] * dm)
    fwd = 2.0 * T * (active + head) + core
    if case["task"] == "eval":
        return {"bytes": 2.0 * (weights + 2 * head), "flops": fwd}
    if case["task"] == "lora":                    # data gradients only; the base weights are read, the adapters trained
        return {"bytes": 2.0 * (weights + 2 * head), "flops": 2 * fwd + core}
    state = {"adamw": 16.0, "adamw16": 8.0, "muon": 4.0}[case["optimizer"]]
    muon = 0.0
    if case["optimizer"] == "muon":               # five Newton-Schulz iterations over each matrix
        f = d["expert_dim"]
        for m, n in [(q, dm), (kv, dm), (kv, dm), (dm, q), (f, dm), (f, dm), (dm, f)]:
            a, b = min(m, n), max(m, n)
            muon += L * 5 * 2.0 * (2 * a * a * b + a * a * a)
    # weights read and written, gradients written, optimizer state read and written (embedding and head: AdamW's)
    moments = 8.0 if case["optimizer"] == "adamw16" else 16.0
    return {"bytes": weights * (6.0 + state) + 2 * head * (6.0 + moments), "flops": 3 * fwd + muon}


def tolerance(case):
    # Four times the distance, on the listed cases, between these kernels and the library's GEMMs and attention in the same
    # model: gradients of bf16 training steps 0.0025 to 0.013, no element off by more than 0.6 of its tensor's root mean
    # square; evaluated losses 0.0005, no token off by more than 0.0025.
    if case["task"] == "eval":
        return {"rel": 0.002, "max": 0.01}
    return {"rel": 0.03, "max": 0.9}

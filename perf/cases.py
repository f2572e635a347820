"""Workloads that users of this package run, for timing and for comparing outputs.

Six kinds, with the sizes of this repository's own benchmarks (`hybrid_bench.SIZES`, `gpt.OPT_SHAPES`, the operator
shapes of `microbench`):

  mlp            the sparse MLP operator on its own, as a host framework calls it per layer
  opt_decode     one lazy-K/V window (16 steps) of the captured sparse decode step of an OPT-shaped decoder
  opt_prompt     the dense prompt pass of the same decoder
  prompt         a prompt through a Ninolorn or Tifosun decoder
  decode         one captured decode step of such a decoder behind a context
  portions       a request whose prompt arrives in portions, through the request pool

Decoders have fewer layers than the named ones, of the real width: every layer costs the same. fp16 for OPT and bf16 for
the other two are the types the models are served in (fp32 is there for comparisons and not listed). Weights are random;
where trained weights have a property that a computation rests on, these have it too: the residual of the sparse decoder
and of the routed one changes slowly from layer to layer, and what a predictor or a router chooses for a token is decided,
not a tie (the sequences of a sparse batch, which share their choices, run tokens of one kind).
"""
from __future__ import annotations

import math

import torch

from dejavu_b200 import ops
from dejavu_b200.generation import InferenceParams, SequencePool, allocate_kv_cache, step, update_graph_cache
from dejavu_b200.gpt import GPTLMHeadModel, apply_sparsity_knobs, opt_config
from dejavu_b200.ninolorn import NinolornForCausalLM
from dejavu_b200.tifosun import TifosunForCausalLM

DEV = "cuda:0"
VOCAB, WINDOW, STREAMS, GLA_RANK = 50272, 1024, 4, 16
EXPERTS, TOP, DIM, ROT, VDIM, RANK = 8, 2, 128, 64, 128, 512
OPT_STEPS, SP_RANK, TOKEN_KINDS = 16, 1000, 16

# name: (width, heads, key/value heads, recurrent heads, feed-forward, OPT heads, OPT feed-forward, OPT neurons, OPT heads in use)
SIZES = {
    "1b": (2048, 16, 4, 8, 5632, 32, 8192, 1024, 12),
    "7b": (4096, 32, 8, 16, 11008, 32, 16384, 2048, 12),
    "66b": (9216, 72, 8, 36, 24576, 72, 36864, 4096, 24),
}


def listed():
    return [
        # one layer's MLP of a small model: what a call costs when there is next to nothing to do
        {"name": "mlp_768", "kind": "mlp", "width": 768, "ffn": 3072, "rows": 384, "batch": 1},
        # the largest MLP of the family, a batch that shares one index list
        {"name": "mlp_12288_batch16", "kind": "mlp", "width": 12288, "ffn": 49152, "rows": 4096, "batch": 16},
        # one interactive user, the sparse decoder's main use
        {"name": "opt_decode_7b", "kind": "opt_decode", "size": "7b", "layers": 8, "batch": 1, "context": 128},
        # the same on the widest model that one GPU holds
        {"name": "opt_decode_66b", "kind": "opt_decode", "size": "66b", "layers": 4, "batch": 1, "context": 128},
        # sequences decoded in lockstep
        {"name": "opt_decode_7b_batch16", "kind": "opt_decode", "size": "7b", "layers": 8, "batch": 16, "context": 128},
        # a long prompt of odd length
        {"name": "opt_prompt_7b", "kind": "opt_prompt", "size": "7b", "layers": 8, "batch": 1, "prompt": 1983},
        # long prompts of the two other designs
        {"name": "ninolorn_prompt_7b", "kind": "prompt", "model": "ninolorn", "size": "7b", "layers": 8, "batch": 1, "prompt": 4096},
        {"name": "tifosun_prompt_7b", "kind": "prompt", "model": "tifosun", "size": "7b", "layers": 8, "batch": 1, "prompt": 4096},
        # a small model that serves a request in portions, beside others: many short launches
        {"name": "ninolorn_portions_1b", "kind": "portions", "model": "ninolorn", "size": "1b", "layers": 12, "prompt": 1000, "portion": 333},
        # one interactive user each
        {"name": "ninolorn_decode_7b", "kind": "decode", "model": "ninolorn", "size": "7b", "layers": 8, "batch": 1, "context": 1100},
        {"name": "tifosun_decode_1b", "kind": "decode", "model": "tifosun", "size": "1b", "layers": 12, "batch": 1, "context": 1100},
        # a batch of users
        {"name": "tifosun_decode_7b_batch8", "kind": "decode", "model": "tifosun", "size": "7b", "layers": 8, "batch": 8, "context": 1100},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    kind = rng.choice(("mlp", "opt_decode", "opt_prompt", "prompt", "decode", "portions"))
    size = rng.choice(("1b", "7b"))
    layers = 2 * rng.randint(1, 6 if size == "1b" else 4)
    model = rng.choice(("ninolorn", "tifosun"))
    if kind == "mlp":
        width = rng.choice((768, 2048, 4096, 5120, 7168, 9216, 12288))
        return {"kind": kind, "width": width, "ffn": 4 * width, "rows": log(width // 16, width // 2), "batch": log(1, 32)}
    if kind == "opt_decode":
        if rng.random() < 0.2:
            size, layers = "66b", rng.randint(2, 4)
        return {"kind": kind, "size": size, "layers": layers, "batch": log(1, 16), "context": log(17, 600)}
    if kind == "opt_prompt":
        return {"kind": kind, "size": size, "layers": layers, "batch": 1, "prompt": log(130, 1983)}
    if kind == "prompt":
        batch = rng.choice((1, 1, 2, 3))
        return {"kind": kind, "model": model, "size": size, "layers": layers, "batch": batch, "prompt": log(130, 4096 // batch)}
    if kind == "decode":
        return {"kind": kind, "model": model, "size": size, "layers": layers, "batch": log(1, 16), "context": log(100, 1500)}
    return {"kind": kind, "model": model, "size": size, "layers": layers, "prompt": log(300, 2000), "portion": log(100, 700)}


# ---- configurations and weights ---------------------------------------------------------------------------------------

def opt_cfg(case):
    D, _, _, _, _, H, F, K, heads = SIZES[case["size"]]
    cfg = opt_config("opt-125m", n_layer=case["layers"], n_embd=D, hidden_size=D, n_head=H, n_inner=F, vocab_size=VOCAB)
    return apply_sparsity_knobs(cfg, K, heads, heads)


def hybrid_cfg(case):
    D, H, G, R, F, *_ = SIZES[case["size"]]
    if case["model"] == "ninolorn":
        rot = {"base": 500000.0, "dims": 128, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
        mlp = {"kind": "dense", "ff": F, "limit": 7.0}
        attention = {"type": "attention", "mlp": mlp, "mixer": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128,
                                                                "scale": 128 ** -0.5, "mask": {"size": WINDOW}, "rot": rot}}
        gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": R, "dim": 128, "vdim": 256, "tau": 16.0}}
        return {"architecture": "Ninolorn", "vocab": VOCAB, "width": D, "streams": STREAMS,
                "layers": [gla, attention] * (case["layers"] // 2), "loop": None, "norm": {"eps": 1e-6}, "logit_softcap": 30.0}
    ff = F // (TOP + 1) // 64 * 64
    moe = {"kind": "moe", "router": {"experts": EXPERTS, "top": TOP}, "expert": {"ff": ff}, "shared": {"ff": ff}}
    memory = {"type": "mlstm", "mlp": moe, "mixer": {"heads": R, "dim": 128, "vdim": 256, "gate_cap": 15.0}}
    latent = {"type": "latent_attention", "mlp": moe,
              "mixer": {"heads": H, "dim": DIM, "rot_dim": ROT, "vdim": VDIM, "kv_rank": RANK, "scale": (DIM + ROT) ** -0.5,
                        "mask": {"size": WINDOW}, "rot": {"base": 10000.0, "dims": ROT}}}
    first = {**memory, "type": "mlstm_2", "mlp": {"kind": "dense", "ff": F}}
    return {"architecture": "Tifosun", "vocab": VOCAB, "width": D, "layers": [first, latent] + [memory, latent] * (case["layers"] // 2 - 1),
            "norm": {"eps": 1e-6}}


class Random:
    """Tensors from one seed, made on the GPU."""

    def __init__(self, seed, dtype):
        self.gen, self.dtype = torch.Generator(device=DEV).manual_seed(seed), dtype

    def normal(self, *shape, std=0.02, mean=0.0, dtype=None):
        x = torch.randn(*shape, generator=self.gen, device=DEV, dtype=dtype or self.dtype).mul_(std)
        return x.add_(mean) if mean else x

    def f32(self, *shape, std=0.1, mean=0.0):
        return self.normal(*shape, std=std, mean=mean, dtype=torch.float32)

    def ids(self, *shape, below=VOCAB):
        return torch.randint(0, below, shape, generator=self.gen, device=DEV)


def opt_weights(case, seed):
    """State dict of the sparse decoder. Tokens are of 16 kinds; a predictor's favourites for a kind are its top choices."""
    cfg, r = opt_cfg(case), Random(seed, torch.float16)
    D, H, F = cfg.hidden_size, cfg.n_head, cfg.n_inner
    unit = torch.nn.functional.normalize
    kinds = unit(r.f32(TOKEN_KINDS, D), dim=1)
    words = r.f32(VOCAB, D, std=0.5).view(-1, TOKEN_KINDS, D).add_(D ** 0.5 * kinds)
    W = {"transformer.embeddings.word_embeddings.weight": words.view(VOCAB, D).half(),
         "transformer.embeddings.position_embeddings.weight": r.normal(cfg.max_position_embeddings, D, std=0.5),
         "transformer.ln_f.weight": r.normal(D, std=0.1, mean=1.0), "transformer.ln_f.bias": r.normal(D)}
    W["lm_head.weight"] = W["transformer.embeddings.word_embeddings.weight"]

    def predictor(out, chosen):
        fc0, fc1 = r.f32(SP_RANK, D, std=0.02), r.f32(out, SP_RANK, std=0.02)
        best = torch.rand(TOKEN_KINDS, out, generator=r.gen, device=DEV).topk(chosen, 1).indices
        hot = torch.zeros(TOKEN_KINDS, out, device=DEV).scatter_(1, best, 1.0)
        return {"fc0.weight": fc0.half(), "fc1.weight": (fc1 + hot.t() @ unit(kinds @ fc0.t(), dim=1)).half()}

    for i in range(cfg.n_layer):
        layer = {"mixer.Wqkv.weight": r.normal(3 * D, D), "mixer.Wqkv.bias": r.normal(3 * D),
                 "mixer.out_proj.weight": r.normal(D, D, std=0.005), "mixer.out_proj.bias": r.normal(D),
                 "mlp.fc1.weight": r.normal(F, D), "mlp.fc1.bias": r.normal(F),
                 "mlp.fc2.weight": r.normal(F, D, std=0.005).t(), "mlp.fc2.bias": r.normal(D)}
        layer.update({f"mixer.sp.{k}": v for k, v in predictor(H, cfg.att_K[0]).items()})
        layer.update({f"mlp.sp.{k}": v for k, v in predictor(F, cfg.mlp_K).items()})
        for norm in ("norm1", "norm2"):
            layer.update({f"{norm}.weight": r.normal(D, std=0.1, mean=1.0), f"{norm}.bias": r.normal(D)})
        W.update({f"transformer.layers.{i}.{k}": v for k, v in layer.items()})
    return W


def hybrid_weights(case, seed):
    """Checkpoint tensors of the other two decoders."""
    cfg, r = hybrid_cfg(case), Random(seed, torch.bfloat16)
    D, W, routers = cfg["width"], {}, []
    routed = case["model"] == "tifosun"
    for i, layer in enumerate(cfg["layers"]):
        mx, mlp, p = layer["mixer"], layer["mlp"], f"l{i}."
        H, dv = mx["heads"], mx["vdim"]
        if layer["type"] == "attention":
            G = mx["kv_heads"]
            t = {"q": r.normal(H * mx["dim"], D), "k": r.normal(G * mx["dim"], D), "v": r.normal(G * dv, D), "sink": r.f32(H, mean=1.0)}
        elif layer["type"] == "latent_attention":
            t = {"q": r.normal(H * (DIM + ROT), D), "dkv": r.normal(RANK + ROT, D), "g": r.normal(H * dv, D),
                 "dkv.norm": r.f32(RANK, mean=1.0), "uk": r.normal(H * DIM, RANK), "uv": r.normal(H * dv, RANK)}
        else:
            t = {"q": r.normal(H * mx["dim"], D), "k": r.normal(H * mx["dim"], D), "v": r.normal(H * dv, D), "g": r.normal(H * dv, D)}
            if layer["type"] == "gla":
                t.update({"a1": r.normal(GLA_RANK, D), "a2": r.f32(H * mx["dim"], GLA_RANK), "a2.b": r.f32(H * mx["dim"], std=0.5, mean=1.0),
                          "norm": r.f32(dv, mean=1.0)})
            else:
                t.update({"i": r.normal(H, D), "f": r.normal(H, D), "i.b": r.f32(H), "f.b": r.f32(H, std=0.5, mean=3.0),
                          "norm": r.f32(H * dv, mean=1.0)})
        t["o"] = r.normal(D, H * dv)
        W.update({f"{p}mix.{k}": v for k, v in t.items()})
        F = mlp.get("ff")
        if mlp["kind"] == "dense":
            W.update({p + "mlp.gate": r.normal(F, D), p + "mlp.up": r.normal(F, D), p + "mlp.down": r.normal(D, F)})
        else:
            F = mlp["expert"]["ff"]
            W[p + "mlp.router"] = r.normal(EXPERTS, D)
            routers.append(W[p + "mlp.router"])
            for e in [f"e{e}" for e in range(EXPERTS)] + ["shared"]:
                W.update({f"{p}mlp.{e}.gate": r.normal(F, D), f"{p}mlp.{e}.up": r.normal(F, D), f"{p}mlp.{e}.down": r.normal(D, F)})
        for q in "12":
            if routed:  # stored as distances from 1; the second norms make sublayers small beside the residual
                W.update({f"{p}norm{q}": r.f32(D), f"{p}norm{q}b": r.f32(D, std=0.05, mean=-0.75)})
            else:
                W.update({f"{p}norm{q}": r.f32(D, mean=1.0), f"{p}hc{q}.in": r.f32(STREAMS, std=0.05, mean=1 / STREAMS),
                          f"{p}hc{q}.out": r.f32(STREAMS, mean=1.0),
                          f"{p}hc{q}.mix": torch.eye(STREAMS, device=DEV) + r.f32(STREAMS, STREAMS, std=0.05)})
    W["final.norm"], W["head"] = r.f32(D, mean=0.0 if routed else 1.0), r.normal(VOCAB, D)
    embed = r.normal(VOCAB, D, std=1.0, dtype=torch.float32)
    for router in routers:  # a token has two experts of its own in every layer
        unit = torch.nn.functional.normalize(router.float(), dim=1)
        first = r.ids(VOCAB, below=EXPERTS)
        embed += 7.0 * unit[first] + 6.0 * unit[(first + 1 + r.ids(VOCAB, below=EXPERTS - 1)) % EXPERTS]
    W["embed"] = embed.to(torch.bfloat16)
    return W


def inputs(case, seed):
    """What arrives at run time, apart from the weights."""
    r = Random(seed + 1, torch.float16)
    kind, B = case["kind"], case.get("batch", 1)
    if kind == "mlp":
        D, F = case["width"], case["ffn"]
        idx = torch.randperm(F, generator=r.gen, device=DEV)[:case["rows"]].sort().values.int()
        return {"x": r.normal(B, D, std=1.0), "W1": r.normal(F, D), "W2t": r.normal(F, D), "b1": r.normal(F), "b2": r.normal(D), "idx": idx}
    if kind == "opt_decode":
        kinds = r.ids(OPT_STEPS, below=TOKEN_KINDS)
        return {"prompt": r.ids(B, case["context"]), "tokens": r.ids(B, OPT_STEPS, below=VOCAB // TOKEN_KINDS) * TOKEN_KINDS + kinds}
    if kind == "decode":
        return {"prompt": r.ids(B, case["context"]), "tokens": r.ids(B, 1)}
    return {"prompt": r.ids(B, case["prompt"])}


# ---- the work -----------------------------------------------------------------------------------------------------------

def hybrid_model(case, seed):
    cls = NinolornForCausalLM if case["model"] == "ninolorn" else TifosunForCausalLM
    return cls(hybrid_cfg(case), device=DEV).eval().load_tensors(hybrid_weights(case, seed))


def opt_model(case, seed):
    model = GPTLMHeadModel(opt_cfg(case), device=DEV, dtype=torch.float16).eval()
    model.load_state_dict(opt_weights(case, seed))
    return model


def new_params(model, batch, n):
    return InferenceParams(max_sequence_len=n, max_batch_size=batch, key_value_memory_dict=allocate_kv_cache(model, batch, n, torch.device(DEV)))


@torch.inference_mode()
def prepare(case, seed):
    kind, s = case["kind"], {"case": case, **inputs(case, seed)}
    if kind == "mlp":
        return s
    model = s["model"] = opt_model(case, seed) if kind.startswith("opt") else hybrid_model(case, seed)
    if kind in ("opt_decode", "decode"):
        B, n = s["prompt"].shape
        steps = s["tokens"].shape[1]
        s["cache"] = cache = update_graph_cache(model, None, B, n, n + steps)
        cache.inference_params.sequence_len_offset = 0
        step(model, cache.inference_params, s["prompt"], logit_rows=[n - 1])
        s["positions"] = torch.arange(n, n + steps, device=DEV).expand(B, steps)
        if kind == "opt_decode":
            s["scores"] = torch.empty(steps, B, 1, VOCAB, dtype=torch.float16, device=DEV)
    elif kind == "portions":
        s["pool"] = SequencePool(model, case["prompt"], torch.device(DEV))
        s["list"] = s["prompt"][0].tolist()
    else:
        s["params"] = new_params(model, case["batch"], case["prompt"])
    return s


def caches(params):
    """All that the caches hold, layer by layer."""
    return [list(c) for _, c in sorted(params.key_value_memory_dict.items())]


@torch.inference_mode()
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mlp":
        return ops.mlp_sparse(s["x"], s["W1"], s["W2t"], s["idx"], s["b1"], s["b2"])
    model = s["model"]
    if kind == "opt_decode":  # scores a given continuation behind the prompt
        cache, (B, n) = s["cache"], s["prompt"].shape
        model.reset_decode_state(n, torch.device(DEV), n + OPT_STEPS, B)
        for t in range(OPT_STEPS):
            s["scores"][t].copy_(cache.run(s["tokens"][:, t:t + 1], s["positions"][:, t:t + 1]))
        return {"logits": s["scores"], "caches": caches(cache.inference_params)}
    if kind == "decode":
        logits = s["cache"].run(s["tokens"], s["positions"])
        return {"logits": logits, "caches": caches(s["cache"].inference_params)}
    if kind == "portions":
        pool, logits = s["pool"], []
        for p in range(0, len(s["list"]), case["portion"]):
            part = s["list"][p:p + case["portion"]]
            logits.append(pool.run("request", part, [len(part) - 1]))
        held = caches(pool.live["request"])
        pool.end("request")
        return {"logits": logits, "caches": held}
    params, n = s["params"], case["prompt"]
    params.sequence_len_offset = 0
    logits = step(model, params, s["prompt"], logit_rows=[n - 1])
    return {"logits": logits, "caches": caches(params)}


def work(case):
    """Weights that a pass uses are read once; caches it reads are read once, what it adds to them written once."""
    kind, B = case["kind"], case.get("batch", 1)
    if kind == "mlp":
        D, K = case["width"], case["rows"]
        return {"bytes": 2 * (2 * K * D + 2 * B * D + K + D) + 4 * K, "flops": 4.0 * B * K * D}
    L = case["layers"]
    D, H, G, R, F, OH, OF, K, heads = SIZES[case["size"]]
    head = VOCAB * D
    if kind == "opt_decode":
        n, hd = case["context"] + OPT_STEPS / 2, D // OH
        dense, sparse = 4 * D * D + 2 * OF * D, 4 * heads * hd * D + 2 * K * D
        predictors = SP_RANK * (2 * D + OH + OF)
        weights = dense + (L - 1) * sparse + (L - 1) * predictors + head  # layer 0 is dense, the last look-ahead unused
        kv = B * 2 * n * hd * (OH + (L - 1) * heads)
        flops = 2.0 * (B * (dense + (L - 1) * sparse + head) + (L - 1) * predictors) + 2.0 * kv
        return {"bytes": OPT_STEPS * (2 * (weights + kv + B * VOCAB)), "flops": OPT_STEPS * flops}
    if kind == "opt_prompt":
        n = case["prompt"]
        weights = L * (4 * D * D + 2 * OF * D)
        return {"bytes": 2 * (weights + head + 2 * L * n * D + VOCAB), "flops": 2.0 * n * weights + 2.0 * head + 2.0 * L * n * n * D}
    n = 1 if kind == "decode" else case["prompt"]
    context = case["context"] if kind == "decode" else 0
    seen = B * (min(context + 1, WINDOW) if kind == "decode" else sum(min(i + 1, WINDOW) for i in range(n)))
    ring, half = min(WINDOW, context + n), L // 2
    if case["model"] == "ninolorn":
        mlp = 3 * F * D
        rec, att = D * R * (2 * 128 + 2 * 256) + D * GLA_RANK + R * 256 * D, D * 128 * (H + 2 * G) + H * 128 * D
        active = distinct = half * (rec + att + 2 * mlp)
        state, row = R * 128 * 256, G * 256
        attention = half * seen * H * 256
    else:
        ff = F // (TOP + 1) // 64 * 64
        expert = 3 * ff * D
        rec = D * R * (2 * 128 + 2 * 256) + 2 * R * D + R * 256 * D
        att = D * (H * (DIM + ROT) + RANK + ROT + H * VDIM) + RANK * H * (DIM + VDIM) + H * VDIM * D
        active = half * (rec + att) + 3 * F * D + (L - 1) * ((TOP + 1) * expert + EXPERTS * D)
        used = EXPERTS * (1 - (1 - TOP / EXPERTS) ** (B * n))
        distinct = half * (rec + att) + 3 * F * D + (L - 1) * ((used + 1) * expert + EXPERTS * D)
        state, row = R * (128 * 256 + 128 + 1), RANK + ROT
        attention = half * seen * H * (DIM + ROT + VDIM)
    recurrence = half * B * n * 2 * R * 128 * 256
    nbytes = 2 * (distinct + head) + 4 * VOCAB * B + half * B * (4 * state * (2 if kind == "decode" else 1) + 2 * row * ring)
    return {"bytes": nbytes, "flops": 2.0 * (B * n * active + B * head + attention + recurrence)}


def tolerance(case):
    """About four times what these cases differ by from the same computation in 64 bits."""
    if case["kind"] == "mlp":
        return {"rel": 1.2e-3}
    return {"rel": 6e-3 if case["kind"].startswith("opt") else 3e-2}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------

def d(x):
    return x.double()


def norm(x, w, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def log_sigmoid(x):
    return torch.clamp(x, max=0) - torch.log1p(torch.exp(-x.abs()))


def causal(q, k, v, scale, window=None, sink=None):
    """q (n, H, dk), k (n, G, dk), v (n, G, dv), positions 0 .. n-1. -> (n, H, dv)"""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(n, device=q.device)
    hidden = i[None, :] > i[:, None]
    if window is not None:
        hidden |= i[None, :] <= i[:, None] - window
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].t() * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :n] @ v[:, h * G // H]
    return out


def in_ring(rows, cap):
    """(n, ...) by position -> (cap, ...): the last `cap` of them at position % cap."""
    n = rows.shape[0]
    ring = torch.zeros(cap, *rows.shape[1:], dtype=rows.dtype, device=rows.device)
    last = torch.arange(max(0, n - cap), n, device=rows.device)
    ring[last % cap] = rows[last]
    return ring


def yarn(rot):
    dims, base, sc = rot["dims"], rot["base"], rot.get("scaling")
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=DEV)
    if not sc:
        return f, 1.0
    lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * sc[w])) / (2 * math.log(base)) for w in ("fast", "slow"))
    lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
    ramp = ((torch.arange(dims // 2, device=DEV).double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def turn(x, rot, pairs):
    """Rotary positions 0 .. n-1 on x (n, heads, dims); neighbours form a pair, or halves."""
    f, amp = yarn(rot)
    a = torch.arange(x.shape[0], device=x.device).double()[:, None, None] * f
    c, s = a.cos() * amp, a.sin() * amp
    u, v = (x[..., 0::2], x[..., 1::2]) if pairs else x.chunk(2, -1)
    r = (u * c - v * s, v * c + u * s)
    return torch.stack(r, -1).flatten(-2) if pairs else torch.cat(r, -1)


def exact_gla(h, W, p, mx):
    H, dk, dv, n = mx["heads"], mx["dim"], mx["vdim"], h.shape[0]
    q, k, v = ((h @ d(W[p + c]).t()).view(n, H, -1) for c in "qkv")
    a = torch.exp(log_sigmoid((h @ d(W[p + "a1"]).t()) @ d(W[p + "a2"]).t() + d(W[p + "a2.b"])) / mx["tau"]).view(n, H, dk, 1)
    q, k, v = q[:, :, None] * dk ** -0.5, k[..., None], v[:, :, None]
    S, o = torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV), torch.empty(n, H, 1, dv, dtype=torch.float64, device=DEV)
    for t in range(n):
        S.mul_(a[t]).addcmul_(k[t], v[t])
        torch.matmul(q[t], S, out=o[t])
    g = h @ d(W[p + "g"]).t()
    y = norm(o.view(n, H, dv), d(W[p + "norm"])).reshape(n, -1) * g * torch.sigmoid(g)
    return y @ d(W[p + "o"]).t(), [S]


def exact_mlstm(h, W, p, mx):
    H, dk, dv, n, cap = mx["heads"], mx["dim"], mx["vdim"], h.shape[0], mx["gate_cap"]
    q, k, v = ((h @ d(W[p + c]).t()).view(n, H, -1) for c in "qkv")
    i, f = (cap * torch.tanh((h @ d(W[p + c]).t() + d(W[p + c + ".b"])) / cap) for c in "if")
    f, m, ms = log_sigmoid(f), torch.zeros(H, dtype=torch.float64, device=DEV), [torch.zeros(H, dtype=torch.float64, device=DEV)]
    for t in range(n):
        m = torch.maximum(f[t] + m, i[t])
        ms.append(m)
    ms = torch.stack(ms)
    keep, add = torch.exp(f + ms[:-1] - ms[1:])[..., None, None], torch.exp(i - ms[1:])[..., None]
    k1 = torch.cat([v, torch.ones(n, H, 1, dtype=v.dtype, device=DEV)], 2)[:, :, None]  # the normaliser is one more value column
    ka, q = (k * add)[..., None], q[:, :, None] * dk ** -0.5
    S, o = torch.zeros(H, dk, dv + 1, dtype=torch.float64, device=DEV), torch.empty(n, H, 1, dv + 1, dtype=torch.float64, device=DEV)
    for t in range(n):
        S.mul_(keep[t]).addcmul_(ka[t], k1[t])
        torch.matmul(q[t], S, out=o[t])
    o = o.view(n, H, dv + 1)
    o = o[..., :dv] / (torch.maximum(o[..., dv].abs(), torch.exp(-ms[1:])) + 1e-6)[..., None]
    y = norm(o, 1.0).reshape(n, -1) * d(W[p + "norm"]) * torch.sigmoid(h @ d(W[p + "g"]).t())
    state = torch.cat([S[..., :dv].reshape(H, -1), S[..., dv], m[:, None], torch.zeros(H, -(dk * dv + dk + 1) % 4, dtype=m.dtype, device=DEV)], 1)
    return y @ d(W[p + "o"]).t(), [state]


def exact_window(h, W, p, mx, cap):
    H, G, n = mx["heads"], mx["kv_heads"], h.shape[0]
    q, k = (turn((h @ d(W[p + c]).t()).view(n, m, -1), mx["rot"], False) for c, m in (("q", H), ("k", G)))
    v = (h @ d(W[p + "v"]).t()).view(n, G, -1)
    o = causal(q, k, v, mx["scale"], mx["mask"]["size"], d(W[p + "sink"])).reshape(n, -1)
    return o @ d(W[p + "o"]).t(), [in_ring(k, cap).transpose(0, 1), in_ring(v, cap).transpose(0, 1)]


def exact_latent(h, W, p, mx, cap):
    H, n = mx["heads"], h.shape[0]
    q = (h @ d(W[p + "q"]).t()).view(n, H, -1)
    q = torch.cat([q[..., :DIM], turn(q[..., DIM:], mx["rot"], True)], -1)
    c = h @ d(W[p + "dkv"]).t()
    c = torch.cat([norm(c[:, :RANK], d(W[p + "dkv.norm"])), turn(c[:, None, RANK:], mx["rot"], True)[:, 0]], 1)
    k, v = ((c[:, :RANK] @ d(W[p + w]).t()).view(n, H, -1) for w in ("uk", "uv"))
    k = torch.cat([k, c[:, None, RANK:].expand(n, H, ROT)], -1)
    o = causal(q, k, v, mx["scale"], mx["mask"]["size"]).reshape(n, -1) * torch.sigmoid(h @ d(W[p + "g"]).t())
    return o @ d(W[p + "o"]).t(), [in_ring(c, cap)]


def gated(h, W, p, limit=None):
    g, u = h @ d(W[p + "gate"]).t(), h @ d(W[p + "up"]).t()
    if limit is None:
        a = g * torch.sigmoid(g) * u
    else:
        g = g.clamp(max=limit)
        a = g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1)
    return a @ d(W[p + "down"]).t()


def exact_mlp(h, W, p, mlp):
    if mlp["kind"] == "dense":
        return gated(h, W, p, mlp.get("limit"))
    w, idx = torch.sigmoid(h @ d(W[p + "router"]).t()).topk(TOP, 1)
    y = gated(h, W, p + "shared.")
    for e in range(EXPERTS):
        t, j = (idx == e).nonzero(as_tuple=True)
        y.index_add_(0, t, gated(w[t, j, None] * h[t], W, f"{p}e{e}."))
    return y


def exact_hybrid(case, W, ids, ends, cap):
    """One sequence from position 0: logits behind the tokens before `ends`, and what the caches hold in the end."""
    cfg, held = hybrid_cfg(case), []
    e = d(W["embed"][ids])
    x = e if case["model"] == "tifosun" else e[:, None].repeat(1, STREAMS, 1)

    def sub(x, q, p, f):
        if case["model"] == "tifosun":
            return x + norm(f(norm(x, 1 + d(W[f"{p}norm{q}"]))), 1 + d(W[f"{p}norm{q}b"]))
        y = f(norm(torch.einsum("nsd,s->nd", x, d(W[f"{p}hc{q}.in"])), d(W[f"{p}norm{q}"])))
        return torch.einsum("nsd,st->ntd", x, d(W[f"{p}hc{q}.mix"])) + y[:, None] * d(W[f"{p}hc{q}.out"])[:, None]

    for i, layer in enumerate(cfg["layers"]):
        p, kind, mx = f"l{i}.", layer["type"], layer["mixer"]

        def mixer(h):
            if kind in ("attention", "latent_attention"):
                y, c = (exact_window if kind == "attention" else exact_latent)(h, W, p + "mix.", mx, cap)
            else:
                y, c = (exact_gla if kind == "gla" else exact_mlstm)(h, W, p + "mix.", mx)
            held.append(c)
            return y

        x = sub(x, "1", p, mixer)
        x = sub(x, "2", p, lambda h: exact_mlp(h, W, p + "mlp.", layer["mlp"]))
    x = x[torch.tensor(ends, device=DEV) - 1]
    if case["model"] == "tifosun":
        return norm(x, 1 + d(W["final.norm"])) @ d(W["head"]).t(), held
    z = norm(x.sum(1), d(W["final.norm"])) @ d(W["head"]).t()
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"]), held


def exact_opt(case, W, prompt, tokens=None):
    """The dense prompt pass, and behind it the sparse steps. Logits (last prompt token, or every step) and the caches."""
    cfg = opt_cfg(case)
    (B, n), T = prompt.shape, 0 if tokens is None else tokens.shape[1]
    L, D, H, eps = cfg.n_layer, cfg.hidden_size, cfg.n_head, cfg.layer_norm_epsilon
    hd = D // H
    keys, values = ([torch.zeros(B, H, n + T, hd, dtype=torch.float64, device=DEV) for _ in range(L)] for _ in range(2))
    tables = [d(W[f"transformer.embeddings.{t}_embeddings.weight"]) for t in ("word", "position")]

    def at(i, name):
        return d(W[f"transformer.layers.{i}.{name}"])

    def ln(x, p):
        return torch.nn.functional.layer_norm(x, (D,), d(W[p + ".weight"]), d(W[p + ".bias"]), eps)

    def lin(x, i, name):
        return x @ at(i, name + ".weight").t() + at(i, name + ".bias")

    def best(x, i, part, k):
        s = (x.sum(0) @ at(i, part + ".sp.fc0.weight").t()) @ at(i, part + ".sp.fc1.weight").t()
        return s.topk(k).indices

    x = tables[0][prompt] + tables[1][:n]
    for i in range(L):
        qkv = lin(ln(x, f"transformer.layers.{i}.norm1"), i, "mixer.Wqkv").view(B, n, 3, H, hd)
        keys[i][:, :, :n], values[i][:, :, :n] = qkv[:, :, 1].transpose(1, 2), qkv[:, :, 2].transpose(1, 2)
        o = torch.stack([causal(*t.unbind(1), hd ** -0.5) for t in qkv])
        x = x + lin(o.reshape(B, n, D), i, "mixer.out_proj")
        x = x + lin(lin(ln(x, f"transformer.layers.{i}.norm2"), i, "mlp.fc1").relu_(), i, "mlp.fc2")
    logits = [ln(x[:, -1:], "transformer.ln_f") @ tables[0].t()] if T == 0 else []
    for t in range(T):
        x, heads, neurons = tables[0][tokens[:, t]] + tables[1][n + t], None, None
        for i in range(L):
            next_heads = best(x, i, "mixer", cfg.att_K[0])
            qkv = lin(ln(x, f"transformer.layers.{i}.norm1"), i, "mixer.Wqkv").view(B, 3, H, hd)
            keys[i][:, :, n + t], values[i][:, :, n + t] = qkv[:, 1], qkv[:, 2]
            s = torch.einsum("bhd,bhkd->bhk", qkv[:, 0] * hd ** -0.5, keys[i][:, :, :n + t + 1]).softmax(-1)
            o = torch.einsum("bhk,bhkd->bhd", s, values[i][:, :, :n + t + 1])
            if heads is not None and t % OPT_STEPS != OPT_STEPS - 1:  # the step that fills the window up takes all heads
                o = o * torch.zeros(H, 1, dtype=o.dtype, device=DEV).index_fill_(0, heads, 1.0)
            x = x + lin(o.reshape(B, D), i, "mixer.out_proj")
            next_neurons = best(x, i, "mlp", cfg.mlp_K)
            h, rows = ln(x, f"transformer.layers.{i}.norm2"), slice(None) if neurons is None else neurons
            w1, w2 = (W[f"transformer.layers.{i}.mlp.{m}.weight"] for m in ("fc1", "fc2"))
            h = (h @ d(w1[rows]).t() + at(i, "mlp.fc1.bias")[rows]).relu_()
            x, heads, neurons = x + h @ d(w2[:, rows]).t() + at(i, "mlp.fc2.bias"), next_heads, next_neurons
        logits.append((ln(x, "transformer.ln_f") @ tables[0].t())[:, None])
    held = [[k.view(B, H, n + T, hd // 8, 8).transpose(2, 3).contiguous(), v] for k, v in zip(keys, values)]
    return {"logits": torch.stack(logits) if T else logits[0], "caches": held}


@torch.inference_mode()
def exact(case, seed):
    kind, s = case["kind"], inputs(case, seed)
    if kind == "mlp":
        rows = s["idx"].long()
        h = (d(s["x"]) @ d(s["W1"][rows]).t() + d(s["b1"][rows])).relu_()
        return h @ d(s["W2t"][rows]) + d(s["b2"])
    if kind.startswith("opt"):
        return exact_opt(case, opt_weights(case, seed), s["prompt"], s.get("tokens"))
    W, ids = hybrid_weights(case, seed), s["prompt"]
    if kind == "decode":
        ids = torch.cat([ids, s["tokens"]], 1)
    B, n = ids.shape
    if B * n > 12000:  # the recurrences go token by token
        return None
    step_ends = [*range(case["portion"], n, case["portion"]), n] if kind == "portions" else [n]
    each = [exact_hybrid(case, W, ids[b], step_ends, min(WINDOW, n)) for b in range(B)]
    logits = torch.stack([z for z, _ in each])
    held = [[torch.stack(c) for c in zip(*layer)] for layer in zip(*(c for _, c in each))]
    return {"logits": [z[None] for z in logits[0]] if kind == "portions" else logits, "caches": held}

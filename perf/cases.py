"""The work this framework is measured on: engine steps of three of its model families and the two kernels of its surface that
hosts call by themselves (latent attention, the sampler), through the public entry points (engine.py, ops.py).

An engine case is ONE step of a serving loop as the step loop issues it: the scheduler has packed the batch (prompts of a
prefill step, or one token of every running sequence behind its cached context), `run` executes it and reads the logits back.
Everything runs in bfloat16: the float32 mode of the registered architectures exists to check a design, not to serve it."""
import json
import math

import numpy as np
import torch

from nano_vllm_rs_b200 import engine as E
from nano_vllm_rs_b200 import ops

BLOCK = 256           # tokens of a cache block, the engine's default
STD = 0.02            # of the built-in architectures' seeded weights
F64 = torch.float64


# ---------------------------------------------------------------------------------------------------------------- the cases
def _engine(model, phase, seqs, tokens, vocab, ragged=0.0, prefix=0, **more):
    return dict({"path": "engine", "model": model, "phase": phase, "seqs": seqs, "tokens": tokens, "ragged": ragged, "prefix": prefix,
                 "vocab": vocab}, **more)


def listed():
    """`tokens`: the longest prompt (prefill) or context (decode, the step's own token included) of the batch; `ragged`: how much
    shorter the others may be; `prefix`: how many leading tokens all prompts share.  Where a step returns the logits of many rows
    the vocabulary is cut to 2048, so that the copy of logits to the host, which a serving loop does not make, stays small."""
    return [
        # one user's chat: a single sequence, where every launch and every weight byte counts
        dict(_engine("qwen3-0.6b", "decode", 1, 300, 151936), name="qwen3-0.6b decode 1"),
        # the headline: 256 concurrent sequences half way through 512 + 512 tokens
        dict(_engine("qwen3-0.6b", "decode", 256, 769, 2048), name="qwen3-0.6b decode 256"),
        # a prefill step of a busy server: prompts of mixed lengths packed together
        dict(_engine("qwen3-0.6b", "prefill", 24, 1021, 151936, 0.95), name="qwen3-0.6b prefill ragged"),
        # a shared system prompt: its blocks are computed once, every other sequence reads them through its table
        dict(_engine("qwen3-0.6b", "prefill", 32, 2300, 2048, 0.08, 2048), name="qwen3-0.6b prefill shared"),
        # long documents at the large model's widths
        dict(_engine("qwen3-8b", "prefill", 2, 4096, 151936), name="qwen3-8b prefill 2x4096"),
        # the hybrid families: a full prefill step, and a decode step of a medium batch
        dict(_engine("talapel", "prefill", 8, 1024, 2048), name="talapel prefill 8x1024"),
        dict(_engine("talapel", "decode", 64, 1024, 2048), name="talapel decode 64"),
        dict(_engine("zudatar", "prefill", 8, 1024, 2048), name="zudatar prefill 8x1024"),
        dict(_engine("zudatar", "decode", 61, 1100, 2048, 0.5), name="zudatar decode 61 ragged"),
        # latent attention by itself: whole prompts, and single tokens behind long contexts
        {"name": "latent prefill 8x1024", "path": "latent", "heads": 16, "seqs": 8, "new": 1024, "context": 1024},
        {"name": "latent decode 32x4001", "path": "latent", "heads": 16, "seqs": 32, "new": 1, "context": 4001},
        # sampling with every option on, for a full batch over the full vocabulary
        {"name": "sample 256x151936", "path": "sample", "rows": 256, "vocab": 151936, "top_k": 50, "top_p": 0.9},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(("qwen decode", "qwen prefill", "qwen shared", "large prefill", "hybrid prefill", "hybrid decode", "latent", "sample"))
    ragged = rng.choice((0.0, 0.3, 0.9))
    if kind == "qwen decode":
        seqs = _log(rng, 1, 256)
        return _engine("qwen3-0.6b", "decode", seqs, _log(rng, 16, min(4000, 256 * 769 // seqs)), 2048 if seqs > 4 else 151936, ragged)
    if kind == "qwen prefill":
        seqs = _log(rng, 1, 64)
        return _engine("qwen3-0.6b", "prefill", seqs, _log(rng, 5, 16000 // seqs), 2048 if seqs > 16 else 151936, ragged)
    if kind == "qwen shared":
        seqs, prefix = _log(rng, 2, 32), BLOCK * rng.randint(1, 8)
        return _engine("qwen3-0.6b", "prefill", seqs, prefix + _log(rng, 16, 300), 2048, 0.0, prefix)
    if kind == "large prefill":
        seqs = _log(rng, 1, 8)
        return _engine("qwen3-8b", "prefill", seqs, _log(rng, 64, 8000 // seqs), 151936, ragged)
    model = rng.choice(("talapel", "zudatar"))
    if kind == "hybrid prefill":
        seqs = _log(rng, 1, 32)
        return _engine(model, "prefill", seqs, _log(rng, 33, 8192 // seqs), 2048, ragged)
    if kind == "hybrid decode":
        return _engine(model, "decode", _log(rng, 1, 64), _log(rng, 33, 1500), 2048, ragged)
    if kind == "latent":
        seqs = _log(rng, 1, 64)
        context = _log(rng, 33, 16384 // seqs if seqs > 2 else 8192)
        new = rng.choice((1, 1, context, max(1, context // 3)))
        return {"path": "latent", "heads": rng.choice((16, 32)), "seqs": seqs, "new": new, "context": context}
    return {"path": "sample", "rows": _log(rng, 1, 256), "vocab": rng.choice((32768, 151936)), "top_k": rng.choice((0, 20, 50)),
            "top_p": rng.choice((0.0, 0.8, 0.95))}


# ------------------------------------------------------------------------------------------------- models and their weights
# The large model runs a quarter of its layers: they are all alike, and the rounding of 36 random layers in bf16 adds up to more
# than a comparison of logits can use.
QWEN = {"qwen3-0.6b": dict(width=1024, ff=3072, layers=28, heads=16, kv=8, dim=128, tied=True),
        "qwen3-8b": dict(width=4096, ff=12288, layers=9, heads=32, kv=8, dim=128, tied=False)}


def talapel_config(vocab):
    """A parallel layer (capped attention beside a state-space mixer, dense feed-forward) and a retention layer with experts."""
    left = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0, "q_temp": {"coef": 0.1, "every": 256}}
    right = {"heads": 64, "groups": 8, "state": 128, "vdim": 64, "conv": 4, "norm_groups": 8}
    ret = {"heads": 16, "dim": 128, "vdim": 128, "rot": {"base": 10000.0, "dims": 128}, "decay": [1.0 - 2.0 ** (-5 - 3 * i / 16) for i in range(16)]}
    return {"architecture": "Talapel", "vocab": vocab, "width": 2048, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "layers": [{"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0},
                        "mlp": {"kind": "dense", "ff": 8192}},
                       {"type": "retention", "mixer": ret,
                        "mlp": {"kind": "moe", "expert": {"ff": 1408}, "router": {"experts": 64, "top": 6}}}]}


def zudatar_config(vocab):
    """Latent attention, the gated delta rule, windowed attention, and latent attention over the first layer's latents."""
    ff = {"kind": "dense", "ff": 8192}
    lat = {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "q_rank": 768, "scale": 128 ** -0.5, "mask": {"size": 512}}
    att = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 512}, "rot": {"base": 10000.0, "dims": 64}}
    dlt = {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}
    return {"architecture": "Zudatar", "vocab": vocab, "width": 2048, "norm": {"eps": 1e-5}, "logit_scale": 1.0,
            "embedding": {"scale": 1.0, "bigram": {"buckets": 4093, "mul_prev": 33, "mul_cur": 5}},
            "layers": [{"type": "latent_attention", "mixer": lat, "mlp": ff}, {"type": "channel_delta", "mixer": dlt, "mlp": None},
                       {"type": "attention", "mixer": att, "mlp": ff}, {"type": "latent_attention", "mixer": dict(lat, kv_from=0), "mlp": ff}]}


CONFIGS = {"talapel": talapel_config, "zudatar": zudatar_config}
LOW_RANK = 128


def _shapes(cfg):
    """The checkpoint's tensors, in a fixed order."""
    W, out = cfg["width"], {"embed": (cfg["vocab"], cfg["width"])}
    if cfg["architecture"] == "Zudatar":
        out["bigram"] = (cfg["embedding"]["bigram"]["buckets"] + 1, W)
    for i, l in enumerate(cfg["layers"]):
        p, q, m, kind = "l%d." % i, "l%d.mix." % i, l["mixer"], l["type"]
        out[p + "norm1"] = (W,)
        if kind == "parallel":
            a, s = m["left"], m["right"]
            H, G, D, V = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            for n, rows in (("q", H * D), ("k", G * D), ("v", G * V)):
                out[q + "left." + n], out[q + "left." + n + ".b"] = (rows, W), (rows,)
            out[q + "left.g"], out[q + "left.o"], out[q + "left.o.b"] = (H * V, W), (W, H * V), (W,)
            inner, gn = s["heads"] * s["vdim"], s["groups"] * s["state"]
            r = q + "right."
            out[r + "in"] = (2 * inner + 2 * gn + s["heads"], W)
            out[r + "conv"], out[r + "conv.b"] = (inner + 2 * gn, s["conv"]), (inner + 2 * gn,)
            out[r + "dt_bias"] = out[r + "A_log"] = out[r + "D"] = (s["heads"],)
            out[r + "norm"], out[r + "o"] = (inner,), (W, inner)
        else:
            H, D, V = m["heads"], m["dim"], m["vdim"]
            if kind == "retention":
                out[q + "q"] = out[q + "k"] = (H * D, W)
                out[q + "v"] = out[q + "g"] = (H * V, W)
            elif kind == "attention":
                out[q + "q"], out[q + "q.b"], out[q + "k"], out[q + "k.b"] = (H * D, W), (H * D,), (m["kv_heads"] * D, W), (m["kv_heads"] * D,)
                out[q + "g"] = (H, W)
            elif kind == "latent_attention":
                out[q + "dq"], out[q + "dq.norm"], out[q + "uq"] = (m["q_rank"], W), (m["q_rank"],), (H * D, m["q_rank"])
                if "kv_from" not in m:
                    out[q + "dkv"], out[q + "dkv.norm"] = (m["kv_rank"], W), (m["kv_rank"],)
                out[q + "uk"], out[q + "uv"], out[q + "sink"], out[q + "g"] = (H * D, m["kv_rank"]), (H * V, m["kv_rank"]), (H,), (H, W)
            else:
                G = m["kv_heads"]
                for n, rows in (("q", G * D), ("k", G * D), ("v", H * V)):
                    out[q + n], out[q + n + ".conv"] = (rows, W), (rows, m["conv"])
                out[q + "b"], out[q + "A_log"], out[q + "norm"] = (H, W), (H,), (V,)
                out[q + "a1"], out[q + "a2"], out[q + "dt_bias"] = (LOW_RANK, W), (H * D, LOW_RANK), (H * D,)
                out[q + "g1"], out[q + "g2"] = (LOW_RANK, W), (H * V, LOW_RANK)
            out[q + "o"] = (W, H * V)
        if cfg["architecture"] == "Zudatar":
            out[p + "norm1b"] = (W,)
        f = l["mlp"]
        if f is None:
            continue
        if cfg["architecture"] == "Zudatar":
            out[p + "norm2"] = out[p + "norm2b"] = (W,)
        if f["kind"] == "dense":
            out[p + "mlp.gate"] = out[p + "mlp.up"] = (f["ff"], W)
            out[p + "mlp.down"] = (W, f["ff"])
        else:
            for e in range(f["router"]["experts"]):
                out[p + "mlp.e%d.up" % e], out[p + "mlp.e%d.down" % e] = (f["expert"]["ff"], W), (W, f["expert"]["ff"])
            out[p + "mlp.table"] = (cfg["vocab"], f["router"]["top"])
    out["final.norm"] = (W,)
    if cfg["architecture"] == "Talapel":
        out["head"] = (cfg["vocab"], W)
    return out


def _checkpoint(cfg, seed):
    """(name, tensor) of every tensor of a registered architecture: matrices keep their rows' scale, norms are near one."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for name, shape in _shapes(cfg).items():
        last = name.split(".")[-1]
        if last == "table":     # `top` different experts for every token
            experts = cfg["layers"][int(name[1:name.index(".")])]["mlp"]["router"]["experts"]
            first = torch.randint(experts, (shape[0], 1), generator=gen, device="cuda")
            yield name, ((first + 11 * torch.arange(shape[1], device="cuda")) % experts).to(torch.int32)
            continue
        x = torch.randn(shape, generator=gen, device="cuda")
        if "norm" in last or last == "D":
            x = 1.0 + 0.2 * x
        elif last in ("A_log", "dt_bias"):
            x = -1.0 + 0.5 * x
        elif last == "b" and len(shape) == 1:
            x = 0.3 * x
        elif last in ("conv", "embed", "bigram"):
            x = 0.5 * x
        elif last != "sink":
            x = x * shape[-1] ** -0.5
        yield name, x.to(torch.bfloat16)


def _lengths(case, rng):
    n, L, lo = case["seqs"], case["tokens"], case["prefix"] + 1
    out = [max(lo, 1, L - int(case["ragged"] * L * u)) for u in rng.random(n)]
    out[0] = L
    return out


def _prompts(case, seed):
    """Token ids of every sequence, the step's own token of a decode case included."""
    rng = np.random.default_rng(seed)
    shared = rng.integers(0, case["vocab"], case["prefix"])
    lens = _lengths(case, rng)
    if case["phase"] == "decode":
        lens = [max(2, n) for n in lens]
    return [np.concatenate([shared, rng.integers(0, case["vocab"], n - case["prefix"])]) for n in lens]


def _prepare_engine(case, seed):
    prompts = _prompts(case, seed)
    decode = case["phase"] == "decode"
    total = sum(len(p) for p in prompts)
    longest = max(len(p) for p in prompts)
    sizes = dict(max_num_seqs=case["seqs"], max_num_batched_tokens=max(longest, min(total, 16384) if decode else total),
                 max_model_len=longest + BLOCK, kvcache_block_size=BLOCK, num_kvcache_blocks=sum(len(p) // BLOCK + 1 for p in prompts) + 1)
    if case["model"] in QWEN:
        eng = E.LLMEngine(E.Config(case["model"], vocab_size=case["vocab"], num_hidden_layers=QWEN[case["model"]]["layers"], **sizes), seed=seed, std=STD)
    else:
        eng = E.LLMEngine(E.Config(model_config=json.dumps(CONFIGS[case["model"]](case["vocab"])), **sizes), init_weights=False)
        for name, t in _checkpoint(CONFIGS[case["model"]](case["vocab"]), seed):
            eng.model_runner.load_weight(name, (t if t.dtype == torch.int32 else t.view(torch.int16)).cpu().numpy().view(
                np.int32 if t.dtype == torch.int32 else np.uint16))
    sp = E.SamplingParams(temperature=0.0, max_tokens=1 << 20, ignore_eos=True)
    at = {eng.add_request(p[:-1] if decode else p, sp): p for p in prompts}
    batch = eng.scheduler.schedule()
    while decode and batch.is_prefill:      # the contexts go through the engine; the next token is the case's own
        eng.model_runner.execute_model(batch)
        eng.scheduler.postprocess([int(at[i][-1]) for i in batch.seq_ids])
        batch = eng.scheduler.schedule()
    return {"path": "engine", "engine": eng, "batch": batch}


# -------------------------------------------------------------------------------------------------- kernels by themselves
RANK, ROT, DIM = 512, 64, 128


def _prepare_latent(case, seed):
    """One layer's folded queries and the cached rows [latent | rotated key part] of every sequence, in scattered blocks."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    H, n, L, new = case["heads"], case["seqs"], case["context"], case["new"]
    per = -(-L // BLOCK)
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    tables = torch.randperm(n * per, generator=gen, device="cuda").to(torch.int32).reshape(n, per)
    cache = randn(n * per * BLOCK, RANK + ROT).to(torch.bfloat16)
    q = randn(n * new, H * (DIM + ROT)).to(torch.bfloat16)
    q_abs = randn(n * new, H * RANK) * (DIM / RANK) ** 0.5      # f32: the folding product keeps its accumulator
    return {"path": "latent", "q": q, "q_abs": q_abs, "cache": cache, "tables": tables, "heads": H,
            "tok_seq": torch.arange(n, device="cuda", dtype=torch.int32).repeat_interleave(new),
            "positions": torch.arange(L - new, L, device="cuda").repeat(n)}


def _prepare_sample(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, V = case["rows"], case["vocab"]
    kinds = torch.rand(n, generator=gen, device="cuda")
    return {"path": "sample", "logits": 2.5 * torch.randn(n, V, generator=gen, device="cuda"),
            "temperatures": torch.where(kinds < 0.125, torch.zeros_like(kinds), 0.5 + kinds),     # some rows are greedy
            "seeds": torch.randint(-(1 << 62), 1 << 62, (n,), generator=gen, device="cuda"),
            "top_k": torch.full((n,), case["top_k"], dtype=torch.int32, device="cuda") if case["top_k"] else None,
            "top_p": torch.full((n,), case["top_p"], device="cuda") if case["top_p"] else None}


def prepare(case, seed):
    return {"engine": _prepare_engine, "latent": _prepare_latent, "sample": _prepare_sample}[case["path"]](case, seed)


def run(state):
    if state["path"] == "engine":
        return state["engine"].model_runner.execute_model(state["batch"], return_logits=True)[1]
    if state["path"] == "latent":
        return ops.latent_attention(state["q_abs"], state["q"], state["tok_seq"], state["positions"], state["tables"], BLOCK, state["cache"],
                                    state["heads"], DIM, ROT, RANK, (DIM + ROT) ** -0.5)
    return ops.sample(state["logits"], state["temperatures"], state["seeds"], state["top_k"], state["top_p"])


# ------------------------------------------------------------------------------------------------------ work and tolerance
def _pairs(case, window=1 << 30):
    """(query, key) pairs of the step under a causal mask, and the keys that it reads (the mean lengths of a ragged batch)."""
    L = case["tokens"] * (1.0 - 0.5 * case["ragged"] * (1.0 - 1.0 / case["seqs"]))
    if case["phase"] == "decode":
        return case["seqs"] * min(L, window), case["seqs"] * min(L, window)
    P = case["prefix"] // BLOCK * BLOCK

    def upto(n):
        w = min(n, window)
        return w * w / 2 + (n - w) * w

    return case["seqs"] * (upto(L) - upto(P)) + upto(P), case["seqs"] * (L - P) + P


def work(case):
    if case["path"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"] + 32.0 * case["rows"], "flops": 2.0 * case["rows"] * case["vocab"]}
    if case["path"] == "latent":
        n, H, L, new = case["seqs"], case["heads"], case["context"], case["new"]
        pairs = n * (new * (L - new) + new * (new + 1) / 2)
        return {"bytes": n * (2.0 * L * (RANK + ROT) + new * H * (4.0 * RANK + 2.0 * ROT + 2.0 * RANK)), "flops": 2.0 * pairs * H * (2 * RANK + ROT)}
    pairs, keys = _pairs(case)
    tokens = case["seqs"] if case["phase"] == "decode" else keys
    logits = case["seqs"] * case["vocab"]
    if case["model"] in QWEN:
        z = QWEN[case["model"]]
        layer = z["width"] * (z["heads"] + 2 * z["kv"]) * z["dim"] + z["heads"] * z["dim"] * z["width"] + 3 * z["width"] * z["ff"]
        kv = 2 * z["kv"] * z["dim"]
        head = z["width"] * case["vocab"]
        return {"bytes": 2.0 * (z["layers"] * (layer + kv * (keys if case["phase"] == "decode" else tokens)) + head) + 4.0 * logits,
                "flops": 2.0 * (z["layers"] * (layer * tokens + 2 * pairs * z["heads"] * z["dim"]) + head * case["seqs"])}
    cfg = CONFIGS[case["model"]](case["vocab"])
    weights = flops = state = 0.0
    for name, shape in _shapes(cfg).items():
        if len(shape) != 2 or name in ("embed", "bigram") or name.endswith("table") or name.endswith("conv"):
            continue
        n = shape[0] * shape[1]
        share, rows = 1.0, case["seqs"] if name == "head" else tokens
        if ".e" in name:      # an expert is read if some token names it, and every token uses `top` of them
            r = cfg["layers"][int(name[1:name.index(".")])]["mlp"]["router"]
            share, rows = 1.0 - (1.0 - r["top"] / r["experts"]) ** min(tokens, case["vocab"]), tokens * r["top"] / r["experts"]
        weights += n * share
        flops += 2.0 * n * rows
    for l in cfg["layers"]:
        m = l["mixer"]
        if l["type"] == "parallel":
            a, s = m["left"], m["right"]
            flops += 2.0 * pairs * a["heads"] * (a["dim"] + a["vdim"]) + 4.0 * tokens * s["heads"] * s["state"] * s["vdim"]
            state += 8.0 * case["seqs"] * s["heads"] * s["state"] * s["vdim"] + 2.0 * keys * a["kv_heads"] * (a["dim"] + a["vdim"])
        elif l["type"] in ("retention", "channel_delta"):
            flops += (4.0 if l["type"] == "retention" else 6.0) * tokens * m["heads"] * m["dim"] * m["vdim"]
            state += 8.0 * case["seqs"] * m["heads"] * m["dim"] * m["vdim"]
        else:
            p, k = _pairs(case, m["mask"]["size"])
            flops += 2.0 * p * m["heads"] * (m["dim"] + m["vdim"])
            state += 2.0 * k * (m["kv_rank"] if l["type"] == "latent_attention" else m["kv_heads"] * 2 * m["dim"])
    if case["model"] == "zudatar":
        weights += cfg["width"] * case["vocab"]
        flops += 2.0 * cfg["width"] * case["vocab"] * case["seqs"]
    return {"bytes": 2.0 * weights + state + 4.0 * logits, "flops": flops}


def tolerance(case):
    if case["path"] == "sample":
        return "exact"
    if case["path"] == "latent":
        return {"rel": 1e-2, "max": 0.2}     # 2.5e-3 from 64 bits: bf16 rows and probabilities
    return {"rel": 0.03, "max": 0.6}         # 0.008 (hybrids) to 0.026 (large model) from 64 bits: bf16 through all layers


# ------------------------------------------------------------------------------------------------------- in 64 bits
def _hashed(count, seed, tensor, start=0):
    """The built-in architectures' seeded weights: four 16-bit fields of a mixed counter, summed, centred and scaled."""
    def signed(x):
        x &= (1 << 64) - 1
        return x - (1 << 64) if x >> 63 else x

    def shifted(x, n):
        return (x >> n) & ((1 << (64 - n)) - 1)

    out = torch.empty(count, dtype=torch.bfloat16, device="cuda")
    for a in range(0, count, 1 << 25):
        b = min(count, a + (1 << 25))
        x = torch.arange(start + a + 1, start + b + 1, device="cuda") * signed(0x9E3779B97F4A7C15) + signed(seed ^ (tensor << 40))
        x = (x ^ shifted(x, 30)) * signed(0xBF58476D1CE4E5B9)
        x = (x ^ shifted(x, 27)) * signed(0x94D049BB133111EB)
        x = x ^ shifted(x, 31)
        s = (x & 0xFFFF) + (shifted(x, 16) & 0xFFFF) + (shifted(x, 32) & 0xFFFF) + shifted(x, 48) - 131070
        out[a:b] = s.to(torch.float32) * (torch.tensor(STD, dtype=torch.float32) * torch.tensor(2.6428998e-05, dtype=torch.float32)).item()
    return out


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(T, dims, base):
    a = torch.arange(T, device="cuda", dtype=F64)[:, None] * base ** (-2.0 * torch.arange(dims // 2, device="cuda", dtype=F64) / dims)
    return a.cos(), a.sin()


def _rotate_half(x, dims, base):
    """x [B, T, heads, dim]: value i of the first `dims` turns with value i + dims / 2."""
    c, s = (t[None, :, None] for t in _angles(x.shape[1], dims, base))
    a, b = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def _rotate_pairs(x, dims, base):
    c, s = (t[None, :, None] for t in _angles(x.shape[1], dims, base))
    a, b = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), x[..., dims:]], -1)


def _attend(q, k, v, scale, window=None, cap=None, sink=None, q_scale=None):
    """Causal attention of [B, T, H, D] queries on [B, T, G, D] keys, one sequence and one block of queries at a time."""
    B, T, H, _ = q.shape
    G = k.shape[2]
    out = torch.empty(B, T, H, v.shape[-1], dtype=F64, device="cuda")
    j = torch.arange(T, device="cuda")
    for b in range(B):
        kb, vb = (t[b].transpose(0, 1).repeat_interleave(H // G, 0) for t in (k, v))
        for lo in range(0, T, 1024):
            hi = min(T, lo + 1024)
            qb = q[b, lo:hi].transpose(0, 1)
            if q_scale is not None:
                qb = qb * q_scale[lo:hi, None]
            s = qb @ kb[:, :hi].transpose(1, 2) * scale
            if cap is not None:
                s = cap * torch.tanh(s / cap)
            hidden = j[None, :hi] > j[lo:hi, None]
            if window is not None:
                hidden = hidden | (j[None, :hi] <= j[lo:hi, None] - window)
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[:, None, None].expand(H, hi - lo, 1)], -1)
            p = torch.softmax(s, -1)
            out[b, lo:hi] = ((p if sink is None else p[..., :-1]) @ vb[:, :hi]).transpose(0, 1)
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _qwen(case, seed, ids, last):
    """ids [B, T] padded; logits at `last`.  A layer's weights are made when it runs."""
    z = QWEN[case["model"]]
    W, D, H, G, eps = z["width"], z["dim"], z["heads"], z["kv"], 1e-6
    mat = lambda t, rows, cols: _hashed(rows * cols, seed, t).reshape(rows, cols).to(F64)
    embed = _hashed(case["vocab"] * W, seed, 1).reshape(-1, W)
    head = embed if z["tied"] else _hashed(case["vocab"] * W, seed, 2).reshape(-1, W)
    group = max(1, 40000 // ids.shape[1])
    parts = [embed[ids[a:a + group]].to(F64) for a in range(0, len(ids), group)]
    for l in range(z["layers"]):
        t = 16 * (l + 1)
        q_w, k_w, v_w = mat(t, H * D, W), mat(t + 1, G * D, W), mat(t + 2, G * D, W)
        o_w, gate, up, down = mat(t + 3, W, H * D), mat(t + 4, z["ff"], W), mat(t + 5, z["ff"], W), mat(t + 6, W, z["ff"])
        for i, x in enumerate(parts):
            h = _rms(x, eps)
            q, k = ((h @ w.T).unflatten(-1, (-1, D)) for w in (q_w, k_w))
            q, k = (_rotate_half(_rms(y, eps), D, 1e6) for y in (q, k))
            x = x + _attend(q, k, (h @ v_w.T).unflatten(-1, (-1, D)), D ** -0.5).flatten(-2) @ o_w.T
            h = _rms(x, eps)
            parts[i] = x + (_silu(h @ gate.T) * (h @ up.T)) @ down.T
            del x, h, q, k
    x = torch.cat([x[torch.arange(len(x), device="cuda"), last[i * group:i * group + len(x)]] for i, x in enumerate(parts)])
    return torch.cat([_rms(x, eps) @ head[a:a + 16384].to(F64).T for a in range(0, case["vocab"], 16384)], -1)


def _conv(x, w, bias=None):
    """Causal convolution of [B, T, channels] over the last `taps` tokens, the last column of w for the token itself."""
    taps = w.shape[1]
    pad = torch.cat([x.new_zeros(x.shape[0], taps - 1, x.shape[2]), x], 1)
    y = sum(pad[:, i:i + x.shape[1]] * w[:, i] for i in range(taps))
    return _silu(y if bias is None else y + bias)


def _scan(decay, k, v, q):
    """S <- decay S + k v^T, y = S^T q; all [B, T, heads, ...], decay [B, T, heads]."""
    S = torch.zeros(*k.shape[:1], *k.shape[2:], v.shape[-1], dtype=F64, device="cuda")
    out = torch.empty_like(v)
    for t in range(k.shape[1]):
        S.mul_(decay[:, t, :, None, None]).add_(k[:, t, ..., None] * v[:, t, :, None])
        out[:, t] = (S * q[:, t, ..., None]).sum(-2)
    return out


def _talapel(w, cfg, ids):
    eps = cfg["norm"]["eps"]
    norm = lambda x, g: torch.nn.functional.layer_norm(x, x.shape[-1:], eps=eps) * g
    x = w["embed"][ids] * cfg["embedding"]["scale"]
    T = ids.shape[1]
    for i, l in enumerate(cfg["layers"]):
        p, q_, m, f = "l%d." % i, "l%d.mix." % i, l["mixer"], l["mlp"]
        h = norm(x, w[p + "norm1"])
        lin = lambda n: h @ w[q_ + n].T
        if l["type"] == "parallel":
            a, s = m["left"], m["right"]
            pos = torch.arange(T, device="cuda", dtype=F64)
            temp = 1.0 + a["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / a["q_temp"]["every"]) + 1.0)
            q, k, v = ((lin("left." + n) + w[q_ + "left.%s.b" % n]).unflatten(-1, (-1, d)) for n, d in (("q", a["dim"]), ("k", a["dim"]), ("v", a["vdim"])))
            y = _attend(q, k, v, a["scale"], cap=a["softcap"], q_scale=temp).flatten(-2)
            mix = m["left_scale"] * ((y * torch.sigmoid(lin("left.g"))) @ w[q_ + "left.o"].T + w[q_ + "left.o.b"])
            inner, gn, heads = s["heads"] * s["vdim"], s["groups"] * s["state"], s["heads"]
            z, xbc, dt = lin("right.in").split([inner, inner + 2 * gn, heads], -1)
            xs, Bm, Cm = _conv(xbc, w[q_ + "right.conv"], w[q_ + "right.conv.b"]).split([inner, gn, gn], -1)
            xs = xs.unflatten(-1, (heads, -1))
            Bm, Cm = (t.unflatten(-1, (s["groups"], -1)).repeat_interleave(heads // s["groups"], 2) for t in (Bm, Cm))
            dt = torch.nn.functional.softplus(dt + w[q_ + "right.dt_bias"])
            y = _scan(torch.exp(-torch.exp(w[q_ + "right.A_log"]) * dt), Bm * dt[..., None], xs, Cm) + w[q_ + "right.D"][:, None] * xs
            y = _rms((y.flatten(-2) * _silu(z)).unflatten(-1, (s["norm_groups"], -1)), eps).flatten(-2) * w[q_ + "right.norm"]
            mix = mix + m["right_scale"] * (y @ w[q_ + "right.o"].T)
        else:
            D = m["dim"]
            q, k, v = (lin(n).unflatten(-1, (m["heads"], -1)) for n in "qkv")
            q, k = (_rotate_half(t, m["rot"]["dims"], m["rot"]["base"]) for t in (q, k))
            decay = torch.tensor(m["decay"], dtype=F64, device="cuda").expand(*ids.shape, -1)
            y = _rms(_scan(decay, k * D ** -0.5, v, q), eps).flatten(-2)
            mix = (y * _silu(lin("g"))) @ w[q_ + "o"].T
        if f["kind"] == "dense":
            mix = mix + (_silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        else:
            flat, names, add = h.reshape(-1, h.shape[-1]), w[p + "mlp.table"][ids.reshape(-1)], torch.zeros_like(h).reshape(-1, h.shape[-1])
            for e in range(f["router"]["experts"]):
                rows = (names == e).any(-1).nonzero()[:, 0]
                add[rows] += torch.relu(flat[rows] @ w[p + "mlp.e%d.up" % e].T).square() @ w[p + "mlp.e%d.down" % e].T / f["router"]["top"]
            mix = mix + add.reshape(h.shape)
        x = x + mix
    return norm(x, w["final.norm"]), w["head"]


def _zudatar(w, cfg, ids):
    eps, bg = cfg["norm"]["eps"], cfg["embedding"]["bigram"]
    rows = torch.cat([torch.full_like(ids[:, :1], bg["buckets"]), (ids[:, :-1] * bg["mul_prev"] + ids[:, 1:] * bg["mul_cur"]) % bg["buckets"]], 1)
    x = w["embed"][ids] * cfg["embedding"]["scale"] + w["bigram"][rows]
    latents = {}
    for i, l in enumerate(cfg["layers"]):
        p, q_, m, f = "l%d." % i, "l%d.mix." % i, l["mixer"], l["mlp"]
        H, D = m["heads"], m["dim"]
        h = _rms(x, eps) * w[p + "norm1"]
        lin = lambda n: h @ w[q_ + n].T
        heads = lambda t: t.unflatten(-1, (-1, D))
        if l["type"] == "attention":
            q, k = heads(lin("q") + w[q_ + "q.b"]), heads(lin("k") + w[q_ + "k.b"])
            turn = lambda t: _rms(_rotate_pairs(t, m["rot"]["dims"], m["rot"]["base"]), eps)
            y = _attend(turn(q), turn(k), k, m["scale"], m["mask"]["size"]) * torch.sigmoid(lin("g"))[..., None]
        elif l["type"] == "latent_attention":
            if "kv_from" not in m:
                latents[i] = _rms(lin("dkv"), eps) * w[q_ + "dkv.norm"]
            c = latents[m.get("kv_from", i)]
            q = heads((_rms(lin("dq"), eps) * w[q_ + "dq.norm"]) @ w[q_ + "uq"].T)
            y = _attend(q, heads(c @ w[q_ + "uk"].T), (c @ w[q_ + "uv"].T).unflatten(-1, (H, -1)), m["scale"], m["mask"]["size"], sink=w[q_ + "sink"])
            y = y * torch.sigmoid(lin("g"))[..., None]
        else:
            q, k, v = (_conv(lin(n), w[q_ + n + ".conv"]).unflatten(-1, (-1, d)) for n, d in (("q", D), ("k", D), ("v", m["vdim"])))
            q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q = q * D ** -0.5
            beta = torch.sigmoid(lin("b"))[..., None]
            dt = heads(torch.nn.functional.softplus(lin("a1") @ w[q_ + "a2"].T + w[q_ + "dt_bias"]))
            g = torch.exp(-torch.exp(w[q_ + "A_log"])[:, None] * dt)
            S = torch.zeros(len(ids), H, D, m["vdim"], dtype=F64, device="cuda")
            y = torch.empty_like(v)
            for t in range(ids.shape[1]):
                S.mul_(g[:, t, ..., None])
                u = beta[:, t] * (v[:, t] - (S * k[:, t, ..., None]).sum(-2))
                S.add_(k[:, t, ..., None] * u[:, :, None])
                y[:, t] = (S * q[:, t, ..., None]).sum(-2)
            y = _rms(y, eps) * w[q_ + "norm"] * torch.sigmoid(lin("g1") @ w[q_ + "g2"].T).unflatten(-1, (H, -1))
        x = x + _rms(y.flatten(-2) @ w[q_ + "o"].T, eps) * w[p + "norm1b"]
        if f is not None:
            h = _rms(x, eps) * w[p + "norm2"]
            x = x + _rms((_silu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T, eps) * w[p + "norm2b"]
    return _rms(x, eps) * w["final.norm"] * cfg["logit_scale"], w["embed"]


def exact(case, seed):
    if case["path"] == "sample":
        return None               # token ids are no computed numbers
    if case["path"] == "latent":
        s = _prepare_latent(case, seed)
        H, n, L, new = case["heads"], case["seqs"], case["context"], case["new"]
        out = torch.empty(n * new, H * RANK, dtype=F64, device="cuda")
        for b in range(n):
            rows = (s["tables"][b].long()[:, None] * BLOCK + torch.arange(BLOCK, device="cuda")).reshape(-1)[:L]
            c = s["cache"][rows].to(F64)
            for lo in range(0, new, 512):
                hi = min(new, lo + 512)
                at = slice(b * new + lo, b * new + hi)
                qa = s["q_abs"][at].to(F64).reshape(-1, H, RANK)
                qr = s["q"][at].to(F64).reshape(-1, H, DIM + ROT)[..., DIM:]
                p = torch.cat([qa, qr], -1) @ c.T * (DIM + ROT) ** -0.5
                p = p.masked_fill((torch.arange(L, device="cuda")[None] > s["positions"][at][:, None])[:, None], -math.inf)
                out[at] = (torch.softmax(p, -1) @ c[:, :RANK]).reshape(-1, H * RANK)
        return out
    prompts = _prompts(case, seed)
    ids = torch.zeros(len(prompts), max(len(p) for p in prompts), dtype=torch.int64)
    for i, p in enumerate(prompts):
        ids[i, :len(p)] = torch.from_numpy(p)
    ids, last = ids.cuda(), torch.tensor([len(p) - 1 for p in prompts], device="cuda")
    if case["model"] in QWEN:
        return _qwen(case, seed, ids, last)
    cfg = CONFIGS[case["model"]](case["vocab"])
    w = {n: t if t.dtype == torch.int32 else t.to(F64) for n, t in _checkpoint(cfg, seed)}
    model = _talapel if case["model"] == "talapel" else _zudatar
    out = []
    for a in range(0, len(ids), 8):
        x, head = model(w, cfg, ids[a:a + 8])
        out.append(x[torch.arange(len(x), device="cuda"), last[a:a + 8]] @ head.T)
    return torch.cat(out)

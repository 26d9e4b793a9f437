"""The work the engine is measured on: serving a set of requests with one of its models.

A pass admits a set of requests, feeds their prompts under a budget of tokens per step while the requests
that are through theirs go on decoding (continuous batching, the way the scheduler packs its steps),
decodes until the last admitted request has its tokens, and gives everything back.  The tokens fed are given ones, as
when a trace is replayed, so that every implementation does the same work whatever its rounding; what comes
back are the fp32 logits of every place that a token would be drawn at.

Sizes are the benchmark's: Llama 3.1 8B, and the models of width 2048 and 4096 with four layers that
``bench.py`` sets beside one another.  Weights are random, with the scales that keep activations of unit size.
"""

from __future__ import annotations

import math

import torch

from mini_infer_b200.engine import ModelRunner, StepEntry

PAGE = 16
BUDGET = 2048          # tokens of a step, the scheduler's default
DEVICE = "cuda:0"

# ------------------------------------------------------------------------------- models

LLAMA_8B = dict(vocab=128256, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, layers=32)
SIZES = {
    2048: dict(heads=16, kv_heads=4, dim=128, window=1024, rot=64, r_heads=4, r_dim=128, r_vdim=256, rank=16,
               unit_width=2560, blocks=10, conv=4, experts=32, top=4, ff=512, shared_ff=1024, vocab=32000,
               chunk=1024, ranks=16, groups=4, keep=2, rot_dim=64, kv_rank=512, dense_ff=5632),
    4096: dict(heads=32, kv_heads=8, dim=128, window=2048, rot=128, r_heads=8, r_dim=128, r_vdim=256, rank=16,
               unit_width=4096, blocks=16, conv=4, experts=64, top=4, ff=1024, shared_ff=2048, vocab=32000,
               chunk=2048, ranks=32, groups=8, keep=4, rot_dim=64, kv_rank=512, dense_ff=11008),
}


def llama_config(width: int) -> dict:
    s = LLAMA_8B if width == 4096 else dict(vocab=32000, width=2048, heads=16, kv_heads=4, dim=128, ff=3072, layers=4)
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": s["vocab"],
            "hidden_size": s["width"], "intermediate_size": s["ff"], "num_hidden_layers": s["layers"],
            "num_attention_heads": s["heads"], "num_key_value_heads": s["kv_heads"], "head_dim": s["dim"],
            "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "max_position_embeddings": 131072,
            "rope_scaling": {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                             "original_max_position_embeddings": 8192},
            "tie_word_embeddings": False}


def ruvurax_config(width: int) -> dict:
    s = SIZES[width]
    mlp = {"kind": "moe", "router": {"experts": s["experts"], "top": s["top"]},
           "expert": {"ff": s["ff"], "limit": 7.0}, "shared": {"ff": s["shared_ff"], "limit": 7.0}}
    unit = {"type": "rglru", "mixer": {"width": s["unit_width"], "blocks": s["blocks"], "conv": s["conv"]}, "mlp": mlp}
    both = {"type": "parallel", "mlp": mlp,
            "mixer": {"left": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": s["dim"], "vdim": s["dim"],
                               "mask": {"size": s["window"]}, "rot": {"base": 10000.0, "dims": s["rot"]},
                               "scale": s["dim"] ** -0.5},
                      "right": {"heads": s["r_heads"], "dim": s["r_dim"], "vdim": s["r_vdim"], "tau": 16.0,
                                "rank": s["rank"]},
                      "left_scale": 1.0, "right_scale": 1.0}}
    return {"architecture": "Ruvurax", "vocab": s["vocab"], "width": width, "embedding": {"scale": 1.0},
            "norm": {"eps": 1e-6}, "layers": [unit, both, unit, both]}


def vepevik_config(width: int) -> dict:
    s = SIZES[width]
    moe = {"kind": "moe", "expert": {"ff": s["ff"]},
           "router": {"experts": s["experts"], "top": s["top"], "scale": 2.5,
                      "groups": {"count": s["groups"], "keep": s["keep"]}}}
    dense = {"kind": "dense", "ff": s["top"] * s["ff"] + s["shared_ff"], "limit": 7.0}
    rot, heads, d = {"base": 10000.0, "dims": s["rot"]}, s["heads"], s["dim"]
    decay = [1.0 - 2.0 ** (-5.0 - 5.0 * h / max(1, heads - 1)) for h in range(heads)]
    ret = {"type": "retention", "mixer": {"heads": heads, "dim": d, "vdim": d, "decay": decay, "rot": rot}}
    att = {"type": "attention", "mixer": {"heads": heads, "kv_heads": s["kv_heads"], "dim": d, "vdim": d,
                                          "mask": {"size": s["chunk"]}, "rot": rot, "scale": d ** -0.5, "v_mix": True}}
    delta = {"type": "channel_delta", "mixer": {"heads": heads, "kv_heads": heads, "dim": d, "vdim": d,
                                                "conv": s["conv"], "ranks": {"decay": s["ranks"], "gate": s["ranks"]}}}
    return {"architecture": "Vepevik", "vocab": s["vocab"], "width": width, "norm": {"eps": 1e-6},
            "layers": [dict(m, mlp=dense if i == 0 else moe) for i, m in enumerate((ret, att, delta, att))]}


def lilulix_config(width: int) -> dict:
    s = SIZES[width]
    mlp = {"kind": "dense", "ff": s["dense_ff"]}
    lat = {"type": "latent_attention", "mlp": mlp,
           "mixer": {"heads": s["heads"], "dim": s["dim"], "rot_dim": s["rot_dim"], "vdim": s["dim"],
                     "kv_rank": s["kv_rank"], "rot": {"base": 10000.0, "dims": s["rot_dim"]},
                     "scale": (s["dim"] + s["rot_dim"]) ** -0.5}}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": s["dim"], "vdim": s["dim"],
                     "scale": s["dim"] ** -0.5}}
    return {"architecture": "Lilulix", "vocab": s["vocab"], "width": width, "norm": {"eps": 1e-6},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 17}},
            "layers": [lat, att, lat, att], "loop": {"start": 1, "stop": 3, "times": 2}}


CONFIGS = {"llama": llama_config, "ruvurax": ruvurax_config, "vepevik": vepevik_config, "lilulix": lilulix_config}


# ------------------------------------------------------------------------------- cases


def listed() -> list[dict]:
    def case(name, model, width, requests, prompt, new, ragged=False, dtype="bfloat16"):
        return {"name": name, "model": model, "width": width, "dtype": dtype, "requests": requests, "prompt": prompt,
                "ragged": ragged, "new": new}

    return [
        # one short question to a small model: launches and latency
        case("llama-2k-turn", "llama", 2048, 1, 17, 16),
        # the float32 engine, with which a conversion or a port is checked
        case("llama-2k-fp32", "llama", 2048, 2, 131, 4, dtype="float32"),
        # the 8B model: one user (the published single-request workload, half as many tokens), a batch of eight with
        # 2048 tokens of context (the benchmark's headline), a busy server with requests of every length, one long document
        case("llama-8b-single", "llama", 4096, 1, 1024, 64),
        case("llama-8b-batch8", "llama", 4096, 8, 2048, 64),
        case("llama-8b-busy", "llama", 4096, 64, 500, 24, ragged=True),
        case("llama-8b-document", "llama", 4096, 1, 8192, 4),
        # recurrent units, linear attention and experts: a long prompt read, and a batch that mostly decodes
        case("ruvurax-2k-prompt", "ruvurax", 2048, 1, 4001, 2),
        case("ruvurax-4k-decode", "ruvurax", 4096, 8, 200, 48, ragged=True),
        # retention, the delta rule, attention in chunks, grouped experts
        case("vepevik-4k-prompt", "vepevik", 4096, 3, 2000, 2, ragged=True),
        case("vepevik-2k-decode", "vepevik", 2048, 8, 100, 64),
        # attention in a latent space and with a distance bias, a looped stretch
        case("lilulix-4k-prompt", "lilulix", 4096, 2, 3000, 2),
        case("lilulix-2k-decode", "lilulix", 2048, 8, 700, 64, ragged=True),
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(cost(c) for c in listed())
    while True:
        model = rng.choice(["llama", "llama", "llama", "ruvurax", "vepevik", "lilulix"])
        width = rng.choice([2048, 4096])
        dtype = "float32" if width == 2048 and rng.random() < 0.15 else "bfloat16"
        case = {"model": model, "width": width, "dtype": dtype, "requests": log_int(1, 64),
                "prompt": log_int(16, 8192), "ragged": rng.random() < 0.5, "new": log_int(2, 64)}
        if dtype == "float32":
            case.update(requests=log_int(1, 8), prompt=log_int(16, 512), new=log_int(2, 16))
        if cost(case) <= most and sum(lengths(case)) <= 20000:
            return case


def lengths(case: dict) -> list[int]:
    """Prompt lengths: all of ``prompt`` tokens, or spread over a factor of sixteen below it."""
    n = case["requests"]
    if not case["ragged"]:
        return [case["prompt"]] * n
    return [max(1, round(case["prompt"] * 16.0 ** -((i * 0.6180339887) % 1.0))) for i in range(n)]


def steps_of(case: dict) -> list[list[tuple[int, int, int, bool]]]:
    """The steps of a pass, each a list of (request, its first token, tokens, whether its last place is wanted)."""
    lens = lengths(case)
    fed, steps = [0] * len(lens), []
    while any(fed[i] < lens[i] + case["new"] for i in range(len(lens))):
        room, step = BUDGET, []
        for i, n in enumerate(lens):
            if fed[i] >= n:
                step.append((i, fed[i], 1, True))
                room -= 1
        for i, n in enumerate(lens):
            take = min(room, n - fed[i])
            if fed[i] < n and take > 0:
                step.append((i, fed[i], take, fed[i] + take == n))
                room -= take
        for i, _, take, _ in step:
            fed[i] += take
        steps.append(step)
    return steps


def total_lengths(case: dict) -> list[int]:
    out = [0] * case["requests"]
    for step in steps_of(case):
        for i, first, n, _ in step:
            out[i] = first + n
    return out


# ------------------------------------------------------------------------------- inputs


class Draw:
    def __init__(self, seed: int, salt: str) -> None:
        self.gen = torch.Generator(device=DEVICE).manual_seed(seed * 1000 + sum(map(ord, salt)))

    def mat(self, *shape, std=None):
        std = std if std is not None else shape[-1] ** -0.5
        return torch.randn(*shape, generator=self.gen, device=DEVICE, dtype=torch.bfloat16).mul_(std)

    def out(self, *shape):
        """A matrix that writes into the stream, scaled down as deep models are initialised."""
        return self.mat(*shape, std=0.35 * shape[-1] ** -0.5)

    def vec(self, n, mean=0.0, std=0.1):
        return (torch.randn(n, generator=self.gen, device=DEVICE) * std + mean).to(torch.bfloat16)


def weights(case: dict, cfg: dict, seed: int) -> dict[str, torch.Tensor]:
    d = Draw(seed, case["model"])
    return {"llama": llama_weights, "ruvurax": ruvurax_weights, "vepevik": vepevik_weights,
            "lilulix": lilulix_weights}[case["model"]](cfg, d)


def llama_weights(cfg: dict, d: Draw) -> dict:
    H, ff, dim = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    nq, nkv, V = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["vocab_size"]
    st = {"model.embed_tokens.weight": d.mat(V, H, std=1.0), "lm_head.weight": d.mat(V, H),
          "model.norm.weight": d.vec(H, 1.0)}
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        st.update({p + "input_layernorm.weight": d.vec(H, 1.0), p + "post_attention_layernorm.weight": d.vec(H, 1.0),
                   a + "q_proj.weight": d.mat(nq * dim, H), a + "k_proj.weight": d.mat(nkv * dim, H),
                   a + "v_proj.weight": d.mat(nkv * dim, H), a + "o_proj.weight": d.mat(H, nq * dim),
                   p + "mlp.gate_proj.weight": d.mat(ff, H), p + "mlp.up_proj.weight": d.mat(ff, H),
                   p + "mlp.down_proj.weight": d.mat(H, ff)})
    return st


def expert_weights(st: dict, p: str, mlp: dict, H: int, d: Draw) -> None:
    E, ff = mlp["router"]["experts"], mlp["expert"]["ff"]
    st[p + "router"] = d.mat(E, H, std=4.0 * H ** -0.5)      # a trained router is decided about most tokens
    for e in range(E):
        st.update({f"{p}e{e}.gate": d.mat(ff, H), f"{p}e{e}.up": d.mat(ff, H), f"{p}e{e}.down": d.out(H, ff)})
    if mlp.get("shared"):
        sf = mlp["shared"]["ff"]
        st.update({p + "shared.gate": d.mat(sf, H), p + "shared.up": d.mat(sf, H), p + "shared.down": d.out(H, sf)})


def ruvurax_weights(cfg: dict, d: Draw) -> dict:
    H = cfg["width"]
    st = {"embed": d.mat(cfg["vocab"], H, std=1.0), "head": d.mat(cfg["vocab"], H),
          "final.norm": d.vec(H, 1.0), "final.norm.b": d.vec(H)}
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        for n in ("norm1", "norm2"):
            st[p + n], st[p + n + ".b"] = d.vec(H, 1.0), d.vec(H)
        q = p + "mix."
        if layer["type"] == "rglru":
            C, B = m["width"], m["blocks"]
            w = C // B
            st.update({q + "y": d.mat(C, H), q + "y.b": d.vec(C), q + "x": d.mat(C, H), q + "x.b": d.vec(C),
                       q + "conv": d.mat(C, m["conv"]), q + "conv.b": d.vec(C),
                       q + "ra": d.mat(B, w, w), q + "ra.b": d.vec(C).reshape(B, w),
                       q + "ri": d.mat(B, w, w), q + "ri.b": d.vec(C).reshape(B, w),
                       q + "lam": d.vec(C, -1.0, 1.0), q + "o": d.out(H, C)})
        else:
            L, R = m["left"], m["right"]
            hk, hv, r = R["heads"] * R["dim"], R["heads"] * R["vdim"], R["rank"]
            st.update({q + "left.q": d.mat(L["heads"] * L["dim"], H), q + "left.k": d.mat(L["kv_heads"] * L["dim"], H),
                       q + "left.v": d.mat(L["kv_heads"] * L["vdim"], H), q + "left.g": d.mat(L["heads"] * L["vdim"], H),
                       q + "left.o": d.out(H, L["heads"] * L["vdim"]),
                       q + "right.q": d.mat(hk, H), q + "right.k": d.mat(hk, H), q + "right.v": d.mat(hv, H),
                       q + "right.g": d.mat(hv, H), q + "right.o": d.out(H, hv), q + "right.norm": d.vec(R["vdim"], 1.0),
                       q + "right.a1": d.mat(r, H), q + "right.a2": d.mat(hk, r), q + "right.a2.b": d.vec(hk, 1.0, 1.0)})
        expert_weights(st, p + "mlp.", layer["mlp"], H, d)
    return st


def vepevik_weights(cfg: dict, d: Draw) -> dict:
    H = cfg["width"]
    st = {"embed": d.mat(cfg["vocab"], H), "embed.norm": d.vec(H, 1.0), "final.norm": d.vec(H, 1.0)}
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        st[p + "norm1"], st[p + "norm2"] = d.vec(H, 1.0), d.vec(H, 1.0)
        q = p + "mix."
        hk, hv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
        if layer["type"] == "retention":
            st.update({q + n: d.mat(r, H) for n, r in (("q", hk), ("k", hk), ("v", hv), ("g", hv))})
        elif layer["type"] == "channel_delta":
            gk, taps, r = m["kv_heads"] * m["dim"], m["conv"], m["ranks"]
            st.update({q + "q": d.mat(gk, H), q + "q.conv": d.mat(gk, taps), q + "k": d.mat(gk, H),
                       q + "k.conv": d.mat(gk, taps), q + "v": d.mat(hv, H), q + "v.conv": d.mat(hv, taps),
                       q + "b": d.mat(m["heads"], H), q + "A_log": d.vec(m["heads"], -0.5, 1.0),
                       q + "norm": d.vec(m["vdim"], 1.0), q + "a1": d.mat(r["decay"], H), q + "a2": d.mat(hk, r["decay"]),
                       q + "dt_bias": d.vec(hk, -1.0, 1.5), q + "g1": d.mat(r["gate"], H), q + "g2": d.mat(hv, r["gate"])})
        else:
            nkv, dim = m["kv_heads"], m["dim"]
            st.update({q + "q": d.mat(hk, H), q + "k": d.mat(nkv * dim, H), q + "v": d.mat(nkv * m["vdim"], H),
                       q + "q.norm": d.vec(dim, 1.0, 0.3), q + "k.norm": d.vec(dim, 1.0, 0.3),
                       q + "g": d.mat(m["heads"], H), q + "vmix": d.vec(1, 0.4).reshape(())})
        st[q + "o"] = d.out(H, hv)
        if mlp["kind"] == "dense":
            st.update({p + "mlp.gate": d.mat(mlp["ff"], H), p + "mlp.up": d.mat(mlp["ff"], H),
                       p + "mlp.down": d.out(H, mlp["ff"])})
        else:
            expert_weights(st, p + "mlp.", mlp, H, d)
    return st


def lilulix_weights(cfg: dict, d: Draw) -> dict:
    H = cfg["width"]
    st = {"embed": d.mat(cfg["vocab"], H), "bigram": d.mat(cfg["embedding"]["bigram"]["buckets"] + 1, H),
          "final.norm": d.vec(H, 1.0), "loop.step": d.mat(cfg["loop"]["times"], H)}
    st["embed"].mul_(16.0)                # the table is the output head as well: between the scales of the two uses
    st["bigram"].mul_(8.0)
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        st[p + "norm1"] = d.vec(H, 1.0)
        q, n = p + "mix.", m["heads"]
        if layer["type"] == "latent_attention":
            R = m["kv_rank"]
            st.update({q + "q": d.mat(n * (m["dim"] + m["rot_dim"]), H), q + "dkv": d.mat(R + m["rot_dim"], H),
                       q + "dkv.norm": d.vec(R, 1.0), q + "uk": d.mat(n * m["dim"], R), q + "uv": d.mat(n * m["vdim"], R),
                       q + "sink": d.vec(n, 0.0, 1.0), q + "g": d.mat(n * m["vdim"], H), q + "o": d.mat(H, n * m["vdim"])})
        else:
            nkv, dim = m["kv_heads"], m["dim"]
            st.update({q + "q": d.mat(n * dim, H), q + "q.b": d.vec(n * dim), q + "k": d.mat(nkv * dim, H),
                       q + "k.b": d.vec(nkv * dim), q + "q.norm": d.vec(dim, 1.0), q + "k.norm": d.vec(dim, 1.0),
                       q + "o": d.mat(H, n * dim)})
        st.update({p + "mlp.gate": d.mat(ff, H), p + "mlp.up": d.mat(ff, H), p + "mlp.down": d.mat(H, ff)})
    return st


def vocab_of(cfg: dict) -> int:
    return cfg.get("vocab") or cfg["vocab_size"]


def token_ids(case: dict, cfg: dict, seed: int) -> list[list[int]]:
    gen = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab_of(cfg), (n,), generator=gen).tolist() for n in total_lengths(case)]


# ------------------------------------------------------------------------------- a pass


def prepare(case: dict, seed: int) -> dict:
    """A loaded engine, with the decode step of the batch captured as before serving, and the requests."""
    cfg = CONFIGS[case["model"]](case["width"])
    n, total = case["requests"], total_lengths(case)
    runner = ModelRunner.from_state_dict(cfg, weights(case, cfg, seed), device=DEVICE, dtype=case["dtype"],
                                         num_blocks=sum(-(-t // PAGE) for t in total) + 2 * n, block_size=PAGE,
                                         max_requests=n, cuda_graph=True)
    ids = token_ids(case, cfg, seed)
    rids = [f"r{i}" for i in range(n)]
    for r in rids:
        runner.add_request(r)
    runner.step([StepEntry(r, [0], [0]) for r in rids])
    for r in rids:
        runner.free_request(r)
    steps = [[(rids[i], ids[i][first:first + k], (k - 1,) if want else ()) for i, first, k, want in step]
             for step in steps_of(case)]
    return {"runner": runner, "rids": rids, "steps": steps,
            "rows": sum(len(w) for step in steps for _, _, w in step)}


def run(state: dict) -> torch.Tensor:
    runner = state["runner"]
    out = torch.empty((state["rows"], runner.vocab_size), dtype=torch.float32, device=runner.device)
    for r in state["rids"]:
        runner.add_request(r)
    row = 0
    for step in state["steps"]:
        logits = runner.step([StepEntry(*entry) for entry in step]).logits
        if len(logits):
            out[row:row + len(logits)].copy_(logits)      # the next step may overwrite them
            row += len(logits)
    for r in state["rids"]:
        runner.free_request(r)
    return out


# ------------------------------------------------------------------------------- what a pass cannot do without


def mixer_numbers(layer: dict, H: int, kv: int, n: int) -> tuple[float, float, float]:
    """(parameters, numbers of cache and state moved, operations beside the products) of a portion of ``n`` tokens that
    ends a context of ``kv``."""
    m = layer["mixer"]

    def softmax_attention(heads, kv_heads, dk, dv, row, lo):
        pairs = sum(min(lo, p) if lo else p for p in (kv - n + 1, kv)) / 2.0 * n
        seen = min(kv, lo + n) if lo else kv
        return row * (seen + n), 2.0 * pairs * heads * (dk + dv)

    if layer["type"] == "rglru":
        C = m["width"]
        return 3 * H * C + 2 * C * (C // m["blocks"]), 2.0 * (m["conv"]) * C, 0.0
    if layer["type"] == "parallel":
        L, R = m["left"], m["right"]
        hk, hv = R["heads"] * R["dim"], R["heads"] * R["vdim"]
        w = H * L["dim"] * (3 * L["heads"] + 2 * L["kv_heads"]) + H * (2 * hk + 3 * hv + R["rank"]) + R["rank"] * hk
        c, f = softmax_attention(L["heads"], L["kv_heads"], L["dim"], L["vdim"], 2 * L["kv_heads"] * L["dim"], L["mask"]["size"])
        return w, c + 4.0 * hk * R["vdim"], f + 4.0 * n * hk * R["vdim"]
    heads, d = m["heads"], m["dim"]
    hd = heads * d
    if layer["type"] == "retention":
        return 5 * H * hd, 4.0 * hd * d, 4.0 * n * hd * d
    if layer["type"] == "channel_delta":
        return 4 * H * hd + H * heads + 2 * m["ranks"]["decay"] * (H + hd), 4.0 * hd * d, 8.0 * n * hd * d
    if layer["type"] == "latent_attention":
        R, r = m["kv_rank"], m["rot_dim"]
        w = H * heads * (d + r) + H * (R + r) + 2 * hd * R + 2 * H * hd
        c, f = softmax_attention(heads, 1, d + r, d, R + r, None)
        return w, c, f
    kvd = m["kv_heads"] * d
    c, f = softmax_attention(heads, m["kv_heads"], d, d, 2 * kvd, (m.get("mask") or {}).get("size"))
    gate = H * heads if "v_mix" in m else 0
    shared = "v_mix" not in m and not layer.get("own_values")         # keys that are the values as well
    return 2 * H * hd + H * kvd * (1 if shared else 2) + gate, c, f


def layer_runs(cfg: dict) -> list[dict]:
    if "hidden_size" in cfg:
        one = {"type": "attention", "own_values": True, "mlp": {"kind": "dense", "ff": cfg["intermediate_size"]},
               "mixer": {"heads": cfg["num_attention_heads"], "kv_heads": cfg["num_key_value_heads"], "dim": cfg["head_dim"]}}
        return [one] * cfg["num_hidden_layers"]
    loop = cfg.get("loop") or {"start": 0, "stop": 0, "times": 1}
    a, b = loop["start"], loop["stop"]
    return cfg["layers"][:a] + cfg["layers"][a:b] * loop["times"] + cfg["layers"][b:]


def work(case: dict) -> dict:
    """Every step reads its weights (of the experts, those its tokens choose in expectation; no chip keeps them between
    steps) and the cache rows and states of its requests, and writes its own; logits are written once."""
    cfg = CONFIGS[case["model"]](case["width"])
    size = 4.0 if case["dtype"] == "float32" else 2.0
    H, V = cfg.get("width") or cfg["hidden_size"], vocab_of(cfg)
    nbytes = flops = 0.0
    for step in steps_of(case):
        tokens = sum(k for _, _, k, _ in step)
        wanted = sum(1 for _, _, _, want in step if want)
        nbytes += size * tokens * H + (size * V * H if wanted else 0.0) + 4.0 * V * wanted
        flops += 2.0 * V * H * wanted
        for layer in layer_runs(cfg):
            params = 0.0
            for _, first, k, _ in step:
                params, moved, ops = mixer_numbers(layer, H, first + k, k)
                nbytes += size * moved
                flops += ops
            mlp = layer["mlp"]
            if mlp["kind"] == "dense":
                read = used = 3.0 * H * mlp["ff"]
            else:
                E, top, ff = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
                own = H * E + 3.0 * H * (mlp["shared"]["ff"] if mlp.get("shared") else 0)
                read = own + E * (1.0 - (1.0 - 1.0 / E) ** (tokens * top)) * 3.0 * H * ff
                used = own + top * 3.0 * H * ff
            nbytes += size * (params + read)
            flops += 2.0 * tokens * (params + used)
    return {"bytes": nbytes, "flops": flops}


def cost(case: dict) -> float:
    w = work(case)
    return max(w["bytes"], w["flops"] / 50.0)


def tolerance(case: dict) -> dict:
    # against exact(): 2e-6 in float32, 4e-3 to 9e-3 in bfloat16 (1.4e-2 where a router was undecided)
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    if case["model"] in ("ruvurax", "vepevik"):
        return {"rel": 0.03, "max": 0.99}      # a token whose router is undecided may go to another expert
    return {"rel": 0.02, "max": 0.3}


# ------------------------------------------------------------------------------- the same in 64 bits


def f64(t: torch.Tensor) -> torch.Tensor:
    return t.to(torch.float64)


def unit_rms(x, eps):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def layer_norm(x, w, b, eps):
    x = x - x.mean(dim=-1, keepdim=True)
    return unit_rms(x, eps) * w + b


def silu(z):
    return z * torch.sigmoid(z)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def turn(x, inv, interleaved=False):
    """``x [T, heads, d]`` rotated by ``position * inv``: pairs of neighbours, or of the two halves of the turned dimensions."""
    half = len(inv)
    ang = (torch.arange(len(x), device=x.device, dtype=torch.float32)[:, None] * inv.float()[None, :]).double()[:, None, :] \
        if inv.dtype == torch.float32 else (torch.arange(len(x), device=x.device)[:, None] * inv[None, :])[:, None, :]
    c, s = ang.cos(), ang.sin()
    out = x.clone()
    a, b = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def frequencies(base, dims, device):
    return float(base) ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=device) / dims)


def llama3_frequencies(cfg, device):
    d, sc = cfg["head_dim"], cfg["rope_scaling"]
    inv = 1.0 / (cfg["rope_theta"] ** (torch.arange(0, d, 2, dtype=torch.float32) / d))
    lo, hi, old, factor = (sc[k] for k in ("low_freq_factor", "high_freq_factor", "original_max_position_embeddings", "factor"))
    wave = 2 * math.pi / inv
    smooth = ((old / wave - lo) / (hi - lo)).clamp(0.0, 1.0)
    return ((1 - smooth) * inv / factor + smooth * inv).to(device)


def attend(q, k, v, scale, window=None, chunk=None, slopes=None, sink=None):
    """Causal softmax attention of one sequence: ``q [T, heads, dk]``, ``k, v [T, kv_heads, ...]``."""
    T, heads, _ = q.shape
    per = heads // k.shape[1]
    at = torch.arange(T, device=q.device)
    out = torch.empty(T, heads, v.shape[-1], dtype=q.dtype, device=q.device)
    rows = max(1, min(T, (1 << 27) // T))
    for lo in range(0, T, rows):
        i, j = at[lo:lo + rows, None], at[None, :lo + rows]
        hidden = j > i
        if window:
            hidden = hidden | (i - j >= window)
        if chunk:
            hidden = hidden | (i // chunk != j // chunk)
        for h in range(heads):
            s = (q[lo:lo + rows, h] @ k[:lo + rows, h // per].T) * scale
            if slopes is not None:
                s = s - slopes[h] * (i - j)
            s = s.masked_fill_(hidden, -math.inf)
            if sink is None:
                p = torch.softmax(s, dim=-1)
            else:
                p = torch.softmax(torch.cat([s, sink[h].expand(len(s), 1)], dim=-1), dim=-1)[:, :-1]
            out[lo:lo + rows, h] = p @ v[:lo + rows, h // per]
    return out


def attend_batched(q, k, v, scale):
    """The same for short sequences without masks beside the causal one, all heads at once."""
    T, heads, _ = q.shape
    per = heads // k.shape[1]
    s = torch.einsum("ihd,jhd->hij", q, k.repeat_interleave(per, dim=1)) * scale
    s = s.masked_fill_(torch.ones(T, T, dtype=torch.bool, device=q.device).triu_(1), -math.inf)
    return torch.einsum("hij,jhd->ihd", torch.softmax(s, dim=-1), v.repeat_interleave(per, dim=1))


def conv(x, w):
    taps = w.shape[1]
    x = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(w[:, j] * x[j:len(x) - (taps - 1 - j)] for j in range(taps))


def experts(h, W, p, mlp, act, choose):
    out = torch.zeros_like(h)
    idx, wts = choose(h @ f64(W[p + "router"]).T, mlp["router"])
    for e in range(mlp["router"]["experts"]):
        rows, place = torch.nonzero(idx == e, as_tuple=True)
        if len(rows):
            x = h[rows]
            y = act(x @ f64(W[f"{p}e{e}.gate"]).T, x @ f64(W[f"{p}e{e}.up"]).T) @ f64(W[f"{p}e{e}.down"]).T
            out.index_add_(0, rows, wts[rows, place, None] * y)
    return out


def clamped(limit):
    def act(g, u):
        g, u = g.clamp(max=limit), u.clamp(min=-limit, max=limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1.0)
    return act


def glu(h, W, p, act):
    return act(h @ f64(W[p + "gate"]).T, h @ f64(W[p + "up"]).T) @ f64(W[p + "down"]).T


def each(parts, f, *tensors):
    """``f`` on every request's rows."""
    return torch.cat([f(*(t[a:b] for t in tensors)) for a, b in parts])


def llama_stream(cfg, W, ids, parts):
    eps, dim = cfg["rms_norm_eps"], cfg["head_dim"]
    inv = llama3_frequencies(cfg, ids.device)
    x = f64(W["model.embed_tokens.weight"][ids])

    def mix(q, k, v):
        q, k, v = turn(q.unflatten(1, (-1, dim)), inv), turn(k.unflatten(1, (-1, dim)), inv), v.unflatten(1, (-1, dim))
        return (attend_batched if len(q) <= 768 else attend)(q, k, v, dim ** -0.5).flatten(1)

    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = unit_rms(x, eps) * f64(W[p + "input_layernorm.weight"])
        q, k, v = (a @ f64(W[f"{p}self_attn.{n}_proj.weight"]).T for n in "qkv")
        x = x + each(parts, mix, q, k, v) @ f64(W[p + "self_attn.o_proj.weight"]).T
        a = unit_rms(x, eps) * f64(W[p + "post_attention_layernorm.weight"])
        x = x + (silu(a @ f64(W[p + "mlp.gate_proj.weight"]).T) * (a @ f64(W[p + "mlp.up_proj.weight"]).T)) \
            @ f64(W[p + "mlp.down_proj.weight"]).T
    return unit_rms(x, eps) * f64(W["model.norm.weight"]), W["lm_head.weight"]


def ruvurax_stream(cfg, W, ids, parts):
    eps = cfg["norm"]["eps"]
    x = f64(W["embed"][ids]) * cfg["embedding"]["scale"]

    def choose(z, router):
        vals, idx = torch.topk(z, router["top"], dim=-1)
        return idx, torch.softmax(vals, dim=-1)

    def unit(h, M, m):
        B, C = m["blocks"], m["width"]
        y = gelu(h @ M("y").T + M("y.b"))
        u = each(parts, lambda t: conv(t, M("conv")) + M("conv.b"), h @ M("x").T + M("x.b"))
        ub = u.unflatten(1, (B, C // B))
        r = torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, M("ra")) + M("ra.b")).flatten(1)
        g = torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, M("ri")) + M("ri.b")).flatten(1)
        log_a = -8.0 * r * torch.nn.functional.softplus(M("lam"))
        a, b = log_a.exp(), torch.sqrt(-torch.expm1(2.0 * log_a)) * g * u

        def walk(a, b):
            S, out = torch.zeros_like(a[0]), torch.empty_like(a)
            for t in range(len(a)):
                S = torch.addcmul(b[t], a[t], S, out=out[t])
            return out
        return (each(parts, walk, a, b) * y) @ M("o").T

    def parallel(h, M, m):
        L, R = m["left"], m["right"]
        inv = frequencies(L["rot"]["base"], L["rot"]["dims"], h.device)
        q, k, v = (h @ M("left." + n).T for n in "qkv")

        def masked(q, k, v):
            q, k = (unit_rms(turn(t.unflatten(1, (-1, L["dim"])), inv, interleaved=True), eps) for t in (q, k))
            return attend(q, k, v.unflatten(1, (-1, L["vdim"])), L["scale"], window=L["mask"]["size"]).flatten(1)
        left = (each(parts, masked, q, k, v) * torch.sigmoid(h @ M("left.g").T)) @ M("left.o").T
        n, dk, dv = R["heads"], R["dim"], R["vdim"]
        alpha = torch.sigmoid((h @ M("right.a1").T) @ M("right.a2").T + M("right.a2.b")) ** (1.0 / R["tau"])
        o = each(parts, linear_walk, (h @ M("right.q").T).unflatten(1, (n, dk)) * dk ** -0.5,
                 (h @ M("right.k").T).unflatten(1, (n, dk)), (h @ M("right.v").T).unflatten(1, (n, dv)),
                 alpha.unflatten(1, (n, dk)))
        o = (unit_rms(o, eps) * M("right.norm")).flatten(1)
        right = (o * silu(h @ M("right.g").T)) @ M("right.o").T
        return m["left_scale"] * left + m["right_scale"] * right

    for i, layer in enumerate(cfg["layers"]):
        def M(n, p=f"l{i}.mix."):
            return f64(W[p + n])
        a = layer_norm(x, f64(W[f"l{i}.norm1"]), f64(W[f"l{i}.norm1.b"]), eps)
        b = layer_norm(x, f64(W[f"l{i}.norm2"]), f64(W[f"l{i}.norm2.b"]), eps)
        mlp = layer["mlp"]
        x = x + (unit if layer["type"] == "rglru" else parallel)(a, M, layer["mixer"]) \
            + experts(b, W, f"l{i}.mlp.", mlp, clamped(mlp["expert"]["limit"]), choose) \
            + glu(b, W, f"l{i}.mlp.shared.", clamped(mlp["shared"]["limit"]))
    return layer_norm(x, f64(W["final.norm"]), f64(W["final.norm.b"]), eps), W["head"]


def linear_walk(q, k, v, alpha):
    S = torch.zeros(*k.shape[1:], v.shape[2], dtype=v.dtype, device=v.device)
    out = torch.empty(*v.shape, dtype=v.dtype, device=v.device)
    for t in range(len(v)):
        S.mul_(alpha[t][:, :, None]).addcmul_(k[t][:, :, None], v[t][:, None, :])
        torch.bmm(q[t][:, None, :], S, out=out[t][:, None, :])
    return out


def delta_walk(q, k, v, g, beta):
    S = torch.zeros(*k.shape[1:], v.shape[2], dtype=v.dtype, device=v.device)
    out = torch.empty(*v.shape, dtype=v.dtype, device=v.device)
    for t in range(len(v)):
        S.mul_(g[t][:, :, None])
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None, :], S)[:, 0])
        S.addcmul_(k[t][:, :, None], u[:, None, :])
        torch.bmm(q[t][:, None, :], S, out=out[t][:, None, :])
    return out


def vepevik_stream(cfg, W, ids, parts):
    eps = cfg["norm"]["eps"]
    x = unit_rms(f64(W["embed"][ids]), eps) * f64(W["embed.norm"])
    first_values = []

    def choose(z, router):
        s = torch.softmax(z, dim=-1)
        n = router["groups"]["count"]
        kept = torch.topk(s.unflatten(1, (n, -1)).amax(dim=-1), router["groups"]["keep"], dim=-1).indices
        allowed = torch.zeros(len(s), n, dtype=torch.bool, device=s.device).scatter_(1, kept, True)
        vals, idx = torch.topk(torch.where(allowed.repeat_interleave(s.shape[1] // n, dim=1), s, -1.0), router["top"], dim=-1)
        return idx, vals / (vals.sum(dim=-1, keepdim=True) + 1e-20) * router["scale"]

    def retention(h, M, m):
        n, d = m["heads"], m["dim"]
        inv = frequencies(m["rot"]["base"], m["rot"]["dims"], h.device)
        decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device)[:, None].expand(n, d)

        def walk(q, k, v):
            q, k = turn(q.unflatten(1, (n, d)), inv), turn(k.unflatten(1, (n, d)), inv) * d ** -0.5
            return linear_walk(q, k, v.unflatten(1, (n, m["vdim"])), decay.expand(len(q), n, d))
        o = unit_rms(each(parts, walk, h @ M("q").T, h @ M("k").T, h @ M("v").T), eps).flatten(1)
        return (o * silu(h @ M("g").T)) @ M("o").T

    def delta(h, M, m):
        n, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (each(parts, lambda t, c=c: silu(conv(t, M(c + ".conv"))), h @ M(c).T) for c in "qkv")
        q, k = (t.unflatten(1, (-1, d)).repeat_interleave(n // m["kv_heads"], dim=1) for t in (q, k))
        q, k = (t * torch.rsqrt((t * t).sum(dim=-1, keepdim=True) + 1e-6) for t in (q, k))
        dt = torch.nn.functional.softplus((h @ M("a1").T) @ M("a2").T + M("dt_bias")).unflatten(1, (n, d))
        g = torch.exp(-torch.exp(M("A_log"))[:, None] * dt)
        o = each(parts, delta_walk, q * d ** -0.5, k, v.unflatten(1, (n, dv)), g, torch.sigmoid(h @ M("b").T))
        return ((unit_rms(o, eps) * M("norm")).flatten(1) * torch.sigmoid((h @ M("g1").T) @ M("g2").T)) @ M("o").T

    def chunked(h, M, m):
        d, dv = m["dim"], m["vdim"]
        inv = frequencies(m["rot"]["base"], m["rot"]["dims"], h.device)
        v = (h @ M("v").T).unflatten(1, (-1, dv))
        if first_values:
            v = (1.0 - M("vmix")) * v + M("vmix") * first_values[0]
        else:
            first_values.append(v)

        def masked(q, k, v):
            q = turn(unit_rms(q.unflatten(1, (-1, d)), eps) * M("q.norm"), inv)
            k = turn(unit_rms(k.unflatten(1, (-1, d)), eps) * M("k.norm"), inv)
            return attend(q, k, v, m["scale"], chunk=m["mask"]["size"])
        o = each(parts, masked, h @ M("q").T, h @ M("k").T, v)
        return (o * torch.sigmoid(h @ M("g").T)[:, :, None]).flatten(1) @ M("o").T

    kinds = {"retention": retention, "channel_delta": delta, "attention": chunked}
    for i, layer in enumerate(cfg["layers"]):
        def M(n, p=f"l{i}.mix."):
            return f64(W[p + n])
        x = x + kinds[layer["type"]](unit_rms(x, eps) * f64(W[f"l{i}.norm1"]), M, layer["mixer"])
        b, mlp = unit_rms(x, eps) * f64(W[f"l{i}.norm2"]), layer["mlp"]
        x = x + (glu(b, W, f"l{i}.mlp.", clamped(mlp["limit"])) if mlp["kind"] == "dense" else
                 experts(b, W, f"l{i}.mlp.", mlp, lambda g, u: silu(g) * u, choose))
    return unit_rms(x, eps) * f64(W["final.norm"]), W["embed"]


def lilulix_stream(cfg, W, ids, parts):
    eps, big, loop = cfg["norm"]["eps"], cfg["embedding"]["bigram"], cfg["loop"]

    def pair_rows(t):
        before = torch.cat([t[:1], t[:-1]])
        rows = (before * big["mul_prev"] + t * big["mul_cur"]) % big["buckets"]
        rows[0] = big["buckets"]
        return rows
    first = f64(W["embed"][ids]) + f64(W["bigram"][each(parts, pair_rows, ids)])

    def latent(h, M, m):
        n, d, r, R = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        inv = frequencies(m["rot"]["base"], m["rot"]["dims"], h.device)
        down = h @ M("dkv").T
        c = unit_rms(down[:, :R], eps) * M("dkv.norm")

        def mix(q, kr, kp, v):
            q = q.unflatten(1, (n, d + r))
            q = torch.cat([q[..., :d], turn(q[..., d:], inv)], dim=-1)
            k = torch.cat([kp.unflatten(1, (n, d)), turn(kr[:, None, :], inv).expand(-1, n, r)], dim=-1)
            return attend(q, k, v.unflatten(1, (n, m["vdim"])), m["scale"], sink=M("sink")).flatten(1)
        o = each(parts, mix, h @ M("q").T, down[:, R:], c @ M("uk").T, c @ M("uv").T)
        return (o * torch.sigmoid(h @ M("g").T)) @ M("o").T

    def biased(h, M, m):
        n, d = m["heads"], m["dim"]
        slopes = [2.0 ** (-8.0 * (i + 1) / n) for i in range(n)]
        zero = torch.zeros(n, dtype=h.dtype, device=h.device)

        def mix(q, k):
            q, k = q.unflatten(1, (n, d)), k.unflatten(1, (-1, d))
            return attend(unit_rms(q, eps) * M("q.norm"), unit_rms(k, eps) * M("k.norm"), k, m["scale"], slopes=slopes,
                          sink=zero).flatten(1)
        return each(parts, mix, h @ M("q").T + M("q.b"), h @ M("k").T + M("k.b")) @ M("o").T

    order = [(i, None) for i in range(loop["start"])]
    for t in range(loop["times"]):
        order += [(i, t if i == loop["start"] else None) for i in range(loop["start"], loop["stop"])]
    order += [(i, None) for i in range(loop["stop"], len(cfg["layers"]))]
    x = first
    for i, turn_no in order:
        def M(n, p=f"l{i}.mix."):
            return f64(W[p + n])
        if turn_no is not None:
            x = x + f64(W["loop.step"])[turn_no] + (first if turn_no else 0.0)
        layer = cfg["layers"][i]
        h = unit_rms(x, eps) * f64(W[f"l{i}.norm1"])
        x = x + (latent if layer["type"] == "latent_attention" else biased)(h, M, layer["mixer"]) \
            + glu(h, W, f"l{i}.mlp.", lambda g, u: gelu(g) * u)
    return unit_rms(x, eps) * f64(W["final.norm"]), W["embed"]


STREAMS = {"llama": llama_stream, "ruvurax": ruvurax_stream, "vepevik": vepevik_stream, "lilulix": lilulix_stream}


@torch.inference_mode()
def exact(case: dict, seed: int):
    """The logits of the whole sequences at the wanted places, in float64."""
    cfg = CONFIGS[case["model"]](case["width"])
    W = weights(case, cfg, seed)
    ids = token_ids(case, cfg, seed)
    starts = [0]
    for t in ids:
        starts.append(starts[-1] + len(t))
    parts = list(zip(starts[:-1], starts[1:]))
    flat = torch.tensor([t for row in ids for t in row], dtype=torch.int64, device=DEVICE)
    z, head = STREAMS[case["model"]](cfg, W, flat, parts)
    want = [starts[i] + first + k - 1 for step in steps_of(case) for i, first, k, wanted in step if wanted]
    z = z[torch.tensor(want, device=DEVICE)]
    del W
    out = torch.empty(len(z), len(head), dtype=torch.float64, device=DEVICE)
    for lo in range(0, len(head), 16384):
        out[:, lo:lo + 16384] = z @ f64(head[lo:lo + 16384]).T
    return out

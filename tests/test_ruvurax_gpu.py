"""The Ruvurax architecture in the engine against the plain implementation (``plain_ruvurax``):
every mechanism alone at the kernel level, then whole models of three small configurations
under every way of cutting the work, in float32 and bfloat16, and greedy generation through the
scheduler.  Weights and inputs are made so that a fault shows: a key that stands out just inside
and just outside a window and at a page's border, states that must be zeroed when a slot is used
again, caches filled with NaN where nothing was written."""

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import plain_ruvurax as P
import trace_util as T
from ruvurax_configs import CONFIGS, DECAY_RANK, PAGE_SIZE, prompt, random_state

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

LENGTHS = {"R": [1, 2, 37, 70], "P": [3, 19, 64, 90, 41], "M": [50, 5, 33, 81]}
# A router logit this close to the first one left out is a close call (bfloat16 activations move a
# logit by about 0.01): the other expert is as good an answer, and through keys, values and states it
# reaches the tokens behind, so a request is compared up to its first close call.  Where only the
# last layer routes, a close call stays in its own row.
CLOSE_CALL = {"float32": 1e-3, "bfloat16": 0.05}
MIN_CHECKED = {"float32": 0.5, "bfloat16": 0.2}
ROW_LOCAL = {"R"}


def ops():
    from mini_infer_b200.csrc import ops as o
    return o


def requests_for(which):
    return {f"r{i}": prompt(CONFIGS[which], n, salt=i) for i, n in enumerate(LENGTHS[which])}


_plain_cache = {}


def plain_for(which):
    """float64 logits of every request, and per request the position of its first close router call."""
    if which not in _plain_cache:
        cfg = CONFIGS[which]
        state = random_state(cfg, seed=11, rank=DECAY_RANK[which])
        logits, margins = {}, {}
        for rid, toks in requests_for(which).items():
            m = []
            logits[rid] = P.ruvurax_forward(state, cfg, toks, torch.float64, margins=m).numpy()
            margins[rid] = torch.stack(m).min(dim=0).values.numpy() if m else np.full(len(toks), np.inf)
        _plain_cache[which] = (state, logits, margins)
    return _plain_cache[which]


def make_runner(which, dtype, steps=None, num_blocks=None, max_requests=4, cuda_graph=False):
    from mini_infer_b200.engine import ModelRunner

    state, _, _ = plain_for(which)
    ps = PAGE_SIZE[which]
    if num_blocks is None:
        num_blocks = T.max_tokens_needed(steps) // ps
    runner = ModelRunner.from_state_dict(CONFIGS[which], state, dtype=dtype, block_size=ps, num_blocks=num_blocks,
                                         max_requests=max_requests, cuda_graph=cuda_graph)
    for st in runner.cache.storage:
        st.fill_(float("nan"))            # a slot that was never written must never be read
    for arena in runner.cache.state_arenas.values():
        arena.fill_(float("nan"))         # a state must be zeroed when its slot is handed out
    return runner


def compare(which, dtype, got):
    _, want, margins = plain_for(which)
    scale = max(float(np.abs(w).max()) for w in want.values())
    tol = T.tolerance(dtype, scale)
    checked = total = 0
    for rid, w in want.items():
        assert got[rid].shape == w.shape
        close = margins[rid] < CLOSE_CALL[dtype]
        if which in ROW_LOCAL:
            keep = np.nonzero(~close)[0]
        else:
            keep = np.arange(int(np.nonzero(close)[0][0]) if close.any() else len(w))
        total += len(w)
        checked += len(keep)
        assert np.isfinite(got[rid]).all(), f"{rid}: non-finite logits"
        bad = T.first_bad(got[rid][keep], w[keep], tol)
        assert bad is None, f"{which} {dtype} {rid}: position {keep[bad]} differs by " \
                            f"{np.abs(got[rid][keep[bad]] - w[keep[bad]]).max():.3g} (bound {float(tol):.3g})"
    assert checked >= MIN_CHECKED[dtype] * total, f"only {checked} of {total} rows were compared"


CUTTINGS = {"whole": T.cut_whole, "last_decoded": T.cut_last_decoded, "portions": T.cut_portions,
            "mixed": T.cut_mixed}


@pytest.mark.parametrize("cutting", list(CUTTINGS))
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("which", ["R", "P", "M"])
def test_engine_matches_plain_under_every_cutting(which, dtype, cutting):
    """Whole prompts, prefill then token-by-token decoding, portions down to two tokens, and mixed
    batches of unequal requests in which slots and pages are freed and used again."""
    requests = requests_for(which)
    steps = CUTTINGS[cutting](requests)
    runner = make_runner(which, dtype, steps)
    got = T.collect(steps, T.replay_in_process(runner, steps), CONFIGS[which]["vocab"])
    runner.cache.check()
    assert runner.cache.num_requests == 0
    for gi, pool in enumerate(runner.cache.pools):
        assert runner.cache.num_free_pages(gi) == pool.num_pages
    compare(which, dtype, got)


@pytest.mark.parametrize("which", ["R", "P", "M"])
def test_float32_logits_do_not_depend_on_the_cutting(which):
    """In float32 every sum runs in an order that depends on the position alone: the logits of a
    position are the same bits whole, in portions, decoded, or beside other requests."""
    requests = requests_for(which)
    results = {}
    for name, cut in CUTTINGS.items():
        steps = cut(requests)
        runner = make_runner(which, "float32", steps)
        results[name] = T.collect(steps, T.replay_in_process(runner, steps), CONFIGS[which]["vocab"])
    for name in ("last_decoded", "portions", "mixed"):
        for rid in requests:
            assert np.array_equal(results[name][rid], results["whole"][rid]), f"{which} {name} {rid}"


def test_long_decoding_past_the_window_and_captured_steps():
    """One short prompt, then 150 tokens one by one (windows of 9 and 40 pass over decoded tokens,
    pages leave the window and come back to the pool), kernel by kernel and as captured graphs."""
    which = "P"
    cfg = CONFIGS[which]
    state, _, _ = plain_for(which)
    toks = prompt(cfg, 156, salt=77)
    m = []
    want = P.ruvurax_forward(state, cfg, toks, torch.float64, margins=m).numpy()
    margin = torch.stack(m).min(dim=0).values.numpy()
    from mini_infer_b200.engine import StepEntry
    for graph in (False, True):
        runner = make_runner(which, "float32", num_blocks=12, cuda_graph=graph)   # 96 slots for 156 tokens
        runner.add_request("a")
        rows = [runner.step([StepEntry("a", toks[:6], list(range(6)))]).logits.cpu().numpy()]
        for t in toks[6:]:
            rows.append(runner.step([StepEntry("a", [t], [0])]).logits.cpu().numpy())
        got = np.concatenate(rows)
        close = np.nonzero(margin < CLOSE_CALL["float32"])[0]
        upto = int(close[0]) if close.size else len(toks)
        assert upto > 100
        tol = T.tolerance("float32", float(np.abs(want).max()))
        assert T.first_bad(got[:upto], want[:upto], tol) is None
        runner.free_request("a")
        runner.cache.check()


def test_greedy_generation_through_the_scheduler():
    """Greedy tokens from the engine's own entry point (scheduler, sampler, cache) equal the plain
    implementation's, fed its own tokens, for several prompts generated together."""
    from mini_infer_b200.engine import ContinuousScheduler, Request
    from mini_infer_b200.sampling import SamplingParams

    which = "M"
    cfg = CONFIGS[which]
    state, _, _ = plain_for(which)
    prompts = [prompt(cfg, n, salt=200 + i) for i, n in enumerate([4, 21, 9])]
    n_new = 12
    runner = make_runner(which, "float32", num_blocks=32)
    sched = ContinuousScheduler(runner, max_concurrent=3, max_tokens_per_step=16)
    results = sched.generate([Request(prompt=p, sampling_params=SamplingParams(), max_tokens=n_new) for p in prompts])
    sched.stop()
    for p, r in zip(prompts, results):
        assert len(r.tokens) == n_new
        seq = list(p)
        for tok in r.tokens:
            logits = P.ruvurax_forward(state, cfg, seq, torch.float64)[-1]
            top2 = torch.topk(logits, 2).values
            if float(top2[0] - top2[1]) > 1e-3:     # the plain choice is not a close call
                assert tok == int(logits.argmax()), f"after {len(seq)} tokens"
            seq.append(tok)
    runner.cache.check()
    assert runner.cache.num_requests == 0


# ----------------------------------------------------------------------------- mechanisms alone


def rnd(*shape, seed, scale=1.0, dtype=torch.float32):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


def ctx_for(q_lens, slots):
    """The part of a step context the state kernels read."""
    starts = np.concatenate([[0], np.cumsum(q_lens)[:-1]]).astype(np.int32)
    i32 = lambda a: torch.tensor(np.asarray(a, dtype=np.int32), device=DEV)
    return SimpleNamespace(q_start=i32(starts), q_len=i32(q_lens), state_slot=i32(slots), n_requests=len(q_lens),
                           decode_only=all(n == 1 for n in q_lens), host_q_len=list(q_lens))


@pytest.mark.parametrize("dtype,bound", [(torch.float32, 2e-6), (torch.bfloat16, 1 / 64)])
def test_layer_norm_pair_with_branch_sum(dtype, bound):
    M, H = 7, 50
    stream = rnd(M, H, seed=1, scale=3.0)
    a1, a2 = rnd(M, H, seed=2, dtype=dtype), rnd(M, H, seed=3, dtype=dtype)
    w = [(rnd(H, seed=4) + 1, rnd(H, seed=5)), (rnd(H, seed=6) + 1, rnd(H, seed=7))]
    r = stream.double() + a1.double() + a2.double()
    s = stream.to(DEV).clone()
    outs = ops().add_layernorm(s, [a1.to(DEV), a2.to(DEV)], [(g.to(DEV), b.to(DEV)) for g, b in w], 1e-5, dtype)
    assert torch.allclose(s.cpu().double(), r, atol=1e-6)          # the stream is updated in place, in fp32
    for out, (g, b) in zip(outs, w):
        want = P.layer_norm(r, g.double(), b.double(), 1e-5)
        assert (out.cpu().double() - want).abs().max() <= bound * max(1.0, want.abs().max())
    rows = torch.tensor([5, 0, 5], dtype=torch.int32, device=DEV)
    before = s.clone()
    out, = ops().add_layernorm(s, [a1.to(DEV)], [(w[0][0].to(DEV), w[0][1].to(DEV))], 1e-5, dtype, rows=rows)
    want = P.layer_norm((before.cpu().double() + a1.double())[[5, 0, 5]], w[0][0].double(), w[0][1].double(), 1e-5)
    assert (out.cpu().double() - want).abs().max() <= bound * max(1.0, want.abs().max())
    assert torch.equal(s, before)                                  # a gathered norm leaves the stream alone


@pytest.mark.parametrize("d,dv,rot", [(24, 16, 8), (10, 14, 6), (64, 64, 64), (7, 3, 2)])
def test_interleaved_rotation_unit_norm_and_store(d, dv, rot):
    """Rotation of pairs (2i, 2i+1) on the first ``rot`` dimensions, unit RMS over the head, and keys
    and values landing where the attention kernel looks for them (checked through attention itself
    in the model tests; here: q and k in place, against the plain functions)."""
    M, nq, nkv = 9, 4, 2
    width = nq * d + nkv * d + nkv * dv + 5          # some columns behind, which must stay untouched
    packed = rnd(M, width, seed=8)
    pos = [0, 1, 2, 3, 100, 101, 4095, 7, 8]
    base = 300.0
    inv = (base ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)).float()
    dev = packed.to(DEV).clone()
    ops().rope_norm_store(dev, 0, nq * d, (nq + nkv) * d, nq, nkv, d, dv,
                          positions=torch.tensor(pos, dtype=torch.int32, device=DEV), inv_freq=inv.to(DEV), rot=rot,
                          unit_norm=True, eps=1e-6)
    got = dev.cpu().double()
    x = packed.double()
    for off, n in ((0, nq), (nq * d, nkv)):
        heads = x[:, off:off + n * d].reshape(M, n, d)
        want = P.unit_rms(P.rotate_interleaved(heads, pos, base, rot), 1e-6).reshape(M, n * d)
        # the angle is an fp32 product: its rounding grows with the position
        bound = 2e-5 + 2e-6 * torch.tensor(pos, dtype=torch.float64)[:, None]
        assert ((got[:, off:off + n * d] - want).abs() <= bound).all()
    assert torch.equal(got[:, (nq + nkv) * d:], x[:, (nq + nkv) * d:])  # values and the rest are not touched


SHORT_CUTS = ({0: 23, 1: 9}, [(1, 2), (2, 1), (7, 0), (1, 1), (3, 5), (9, 0)])
LONG_CUTS = ({0: 331, 1: 70}, [(130, 65), (1, 0), (200, 5)])     # long portions: chunks walked side by side


@pytest.mark.parametrize("dtype,bound,plan", [(torch.float32, 1e-5, SHORT_CUTS), (torch.bfloat16, 2e-2, SHORT_CUTS),
                                              (torch.float32, 1e-5, LONG_CUTS), (torch.bfloat16, 2e-2, LONG_CUTS)])
def test_recurrent_unit_carries_its_state_across_portions(dtype, bound, plan):
    """Convolution tail and recurrent state through portions of 1, 2 and more tokens, two requests
    in one launch, against the plain recurrence over the whole sequence."""
    C, blocks, taps, H = 24, 3, 4, 16
    bw = C // blocks
    total, cuts = plan
    W = {"y": rnd(C, H, seed=20, scale=0.3), "y.b": rnd(C, seed=21, scale=0.1), "x": rnd(C, H, seed=22, scale=0.3),
         "x.b": rnd(C, seed=23, scale=0.1), "conv": rnd(C, taps, seed=24, scale=0.5), "conv.b": rnd(C, seed=25, scale=0.1),
         "ra": rnd(blocks, bw, bw, seed=26, scale=0.4), "ra.b": rnd(blocks, bw, seed=27, scale=0.1),
         "ri": rnd(blocks, bw, bw, seed=28, scale=0.4), "ri.b": rnd(blocks, bw, seed=29, scale=0.1),
         "lam": rnd(C, seed=30) - 1.0, "o": torch.eye(C)}
    W = {k: v.to(dtype).float() for k, v in W.items()}
    hs = {r: rnd(n, H, seed=40 + r).to(dtype).float() for r, n in total.items()}
    want = {r: P.rglru_mixer(hs[r].double(), {k: v.double() for k, v in W.items()}, blocks) for r in total}
    state = torch.full((4, taps, C), float("nan"), device=DEV)
    slots = {0: 2, 1: 0}
    for s in slots.values():
        state[s].zero_()
    gates_w = torch.cat([W["ra"], W["ri"]], dim=1).to(dtype).to(DEV).contiguous()
    f32 = lambda t: t.float().to(DEV).contiguous()
    done = {0: 0, 1: 0}
    got = {r: [] for r in total}
    for n0, n1 in cuts:
        lens = [n for n in (n0, n1) if n]
        who = [r for r, n in ((0, n0), (1, n1)) if n]
        h = torch.cat([hs[r][done[r]:done[r] + n] for r, n in zip(who, lens)])
        proj = (h.double() @ torch.cat([W["y"], W["x"]]).double().T).to(dtype).to(DEV)     # [M, 2C]
        ctx = ctx_for(lens, [slots[r] for r in who])
        y, x = proj[:, :C], proj[:, C:]
        u = torch.empty((h.shape[0], C), dtype=dtype, device=DEV)
        ops().causal_conv(x, f32(W["x.b"]), f32(W["conv"]), f32(W["conv.b"]), state, ctx, u)
        gates = ops().block_diagonal_gates(u, gates_w)
        out = torch.empty_like(u)
        ops().rglru_scan(gates, f32(W["ra.b"]).reshape(-1), f32(W["ri.b"]).reshape(-1), f32(W["lam"]), 8.0, u, y,
                         f32(W["y.b"]), x, f32(W["x.b"]), taps, state, ctx, out)
        row = 0
        for r, n in zip(who, lens):
            got[r].append(out[row:row + n].cpu().double())
            row += n
            done[r] += n
    for r in total:
        assert done[r] == total[r]
        g = torch.cat(got[r])
        assert (g - want[r]).abs().max() <= bound * max(1.0, want[r].abs().max()), f"request {r}"
    assert torch.isnan(state[1]).all() and torch.isnan(state[3]).all()      # other slots are never touched


@pytest.mark.parametrize("heads,dk,dv,dtype,portions", [
    (2, 12, 36, torch.float32, (1, 17, 2, 1, 1, 20, 3)), (1, 64, 32, torch.float32, (1, 17, 2, 1, 1, 20, 3)),
    (3, 9, 5, torch.float32, (1, 17, 2, 1, 1, 20, 3)),
    (2, 24, 40, torch.bfloat16, (300, 1, 140, 129)), (1, 128, 64, torch.bfloat16, (513,))])   # chunks side by side
def test_gated_linear_attention_state(heads, dk, dv, dtype, portions):
    """The matrix state through portions and decoded tokens against the plain token loop, with decays
    near 1 and near 0, and a head's output norm and gate."""
    Tn, tau = sum(portions), 3.0
    stride = heads * (2 * dk + dv) + 3
    stride += (-stride) % 8
    packed = rnd(Tn, stride, seed=50).to(dtype)
    z = rnd(Tn, heads * dk, seed=51, scale=3.0)
    zb = rnd(heads * dk, seed=52)
    q, k = packed[:, :heads * dk], packed[:, heads * dk:2 * heads * dk]
    v = packed[:, 2 * heads * dk:2 * heads * dk + heads * dv]
    alpha = torch.sigmoid((z + zb).double()) ** (1.0 / tau)
    S = torch.zeros(heads, dk, dv, dtype=torch.float64)
    want = torch.empty(Tn, heads, dv, dtype=torch.float64)
    for t in range(Tn):
        kt, vt = k[t].double().reshape(heads, dk), v[t].double().reshape(heads, dv)
        S = alpha[t].reshape(heads, dk)[:, :, None] * S + kt[:, :, None] * vt[:, None, :]
        want[t] = torch.einsum("hkv,hk->hv", S, q[t].double().reshape(heads, dk) * dk ** -0.5)
    state = torch.full((3, heads, dk, dv), float("nan"), device=DEV)
    state[1].zero_()
    dev = packed.to(DEV)
    got, t0 = [], 0
    for n in portions:
        ctx = ctx_for([n], [1])
        sl = dev[t0:t0 + n]
        o = ops().gla_scan(sl[:, :heads * dk], sl[:, heads * dk:2 * heads * dk],
                           sl[:, 2 * heads * dk:2 * heads * dk + heads * dv], z[t0:t0 + n].to(DEV).contiguous(),
                           zb.to(DEV), tau, dk ** -0.5, heads, dk, dv, state, ctx)
        got.append(o.cpu().double())
        t0 += n
    got = torch.cat(got).reshape(Tn, heads, dv)
    assert (got - want).abs().max() <= 2e-5 * max(1.0, want.abs().max())
    assert (state[1].cpu().double() - S).abs().max() <= 2e-5 * max(1.0, S.abs().max())
    gain, gate = rnd(dv, seed=53) + 1, rnd(Tn, heads * dv, seed=54)
    out = torch.empty(Tn, heads * dv, device=DEV)
    ops().headnorm_gate(got.reshape(Tn, heads * dv).float().to(DEV), gain.to(DEV), gate.to(DEV), out, heads, dv, 1e-5,
                        "silu", 0.7)
    ref = (P.unit_rms(got, 1e-5) * gain.double()).reshape(Tn, heads * dv) * torch.nn.functional.silu(gate.double()) * 0.7
    assert (out.cpu().double() - ref).abs().max() <= 1e-5 * max(1.0, ref.abs().max())


@pytest.mark.parametrize("heads,dk,dv,portions", [(2, 128, 128, (64, 33, 65)), (1, 130, 129, (200,)), (2, 16, 8, (127, 1, 128)),
                                                  (1, 256, 40, (70, 64))])
@pytest.mark.parametrize("decays", ["slow", "steep", "dead", "head"])
def test_linear_attention_in_chunks(heads, dk, dv, portions, decays):
    """Portions taken as products per 64 tokens at the edges of the chunks and of the 128-wide tiles, with decays that stay
    near 1, that fall by e^-100 within a chunk, that are exactly 0 now and then, and one per head, against the token loop
    in float64.  The error of a sum of products in fp32 is bounded by the number of roundings on the way (64 within a
    chunk, dk + 64 for the sums, a few per chunk) times 2^-24 of the sum of the terms' magnitudes."""
    Tn = sum(portions)
    q, k, v = rnd(Tn, heads * dk, seed=70).bfloat16(), rnd(Tn, heads * dk, seed=71).bfloat16(), rnd(Tn, heads * dv, seed=72).bfloat16()
    z = rnd(Tn, heads * dk, seed=73, scale={"slow": 1.0, "steep": 12.0, "dead": 1.0, "head": 1.0}[decays])
    if decays == "dead":
        z[::7] = -1e4
    per_head = torch.tensor([0.97, 0.2][:heads]) if decays == "head" else None
    alpha = torch.sigmoid(z.double()).reshape(Tn, heads, dk) if per_head is None else per_head.double()[None, :, None].expand(Tn, heads, dk)
    S = torch.zeros(heads, dk, dv, dtype=torch.float64)
    size, want, terms = S.clone(), torch.empty(Tn, heads, dv, dtype=torch.float64), torch.empty(Tn, heads, dv, dtype=torch.float64)
    for t in range(Tn):
        qt, kt, vt = (x[t].double().reshape(heads, -1) for x in (q, k, v))
        S = alpha[t][:, :, None] * S + kt[:, :, None] * vt[:, None, :]
        size = alpha[t][:, :, None] * size + (kt[:, :, None] * vt[:, None, :]).abs()
        want[t], terms[t] = torch.einsum("hkv,hk->hv", S, qt), torch.einsum("hkv,hk->hv", size, qt.abs())
    state = torch.zeros(2, heads, dk, dv, device=DEV)
    got, t0 = [], 0
    for n in portions:
        part = [x[t0:t0 + n].to(DEV) for x in (q, k, v)]
        got.append(ops().gla_scan(*part, None if per_head is not None else z[t0:t0 + n].to(DEV).contiguous(), None, 1.0, 1.0,
                                  heads, dk, dv, state, ctx_for([n], [1]),
                                  head_decay=per_head.to(DEV) if per_head is not None else None).cpu().double())
        t0 += n
    rounds = 64 + (dk + 64) + 4 * (Tn // 64 + 1)
    assert ((torch.cat(got).reshape(Tn, heads, dv) - want).abs() <= rounds * 2.0 ** -24 * terms + 1e-30).all()
    assert ((state[1].cpu().double() - S).abs() <= rounds * 2.0 ** -24 * size + 1e-30).all()


@pytest.mark.parametrize("heads,dk,dv", [(3, 128, 128), (2, 64, 200), (2, 200, 64)])
@pytest.mark.parametrize("decays", ["channel", "head", "token", "token_dead", "steep"])
def test_chunks_are_no_further_from_64_bits_than_the_walk(heads, dk, dv, decays, monkeypatch):
    """800 tokens, every one rounded once per state element in the walk, with decays near 1 (per channel as gates of
    temperature 16 give them, fixed ones, one per token, some of these 0) and steep ones.  Products over 64 tokens carry the roundings
    of their decays to every element and take longer sums: neither may show.  (The state's chain of 64 products is allowed 5
    parts in a hundred: two of its terms' factors are rounded where the walk rounds one.)"""
    o, n = ops(), 800
    q, k, v = rnd(n, heads * dk, seed=70).bfloat16(), rnd(n, heads * dk, seed=71, scale=dk ** -0.5).bfloat16(), rnd(n, heads * dv, seed=72).bfloat16()
    z = rnd(n, heads * dk, seed=73) + 1 if decays == "channel" else rnd(n, heads * dk, seed=73) * 3 - 2 if decays == "steep" else None
    tau = 16.0 if decays == "channel" else 1.0
    hd = torch.tensor([0.96875, 0.99, 0.999][:heads]) if decays == "head" else None
    tg = None
    if decays.startswith("token"):
        tg = torch.stack([torch.sigmoid(rnd(n, heads, seed=74) + 3), torch.sigmoid(rnd(n, heads, seed=75)), torch.zeros(n, heads)], dim=-1)
        if decays == "token_dead":
            tg[::23, :, 0] = 0.0
    alpha = (torch.sigmoid(z.double()).reshape(n, heads, dk) ** (1 / tau) if z is not None else
             hd.double()[None, :, None].expand(n, heads, dk) if hd is not None else tg[..., :1].double().expand(n, heads, dk))
    kk = k.double().reshape(n, heads, dk) * (tg[..., 1:2].double() if tg is not None else 1.0)
    S, want = torch.zeros(heads, dk, dv, dtype=torch.float64), torch.empty(n, heads * dv, dtype=torch.float64)
    for t in range(n):
        S = alpha[t][:, :, None] * S + kk[t][:, :, None] * v[t].double().reshape(heads, 1, dv)
        want[t] = torch.einsum("hkv,hk->hv", S, q[t].double().reshape(heads, dk)).flatten()
    dev = lambda x: None if x is None else x.contiguous().to(DEV)
    off = {}
    for form, limit in (("walk", n), ("chunks", 0)):
        monkeypatch.setattr(o, "GLA_LONG", limit)
        state = torch.zeros(1, heads, dk, dv, device=DEV)
        out = o.gla_scan(dev(q), dev(k), dev(v), dev(z), None, tau, 1.0, heads, dk, dv, state, ctx_for([n], [0]), head_decay=dev(hd),
                         tok_gates=dev(tg))
        off[form] = float((out.cpu().double() - want).norm()), float((state[0].cpu().double() - S).norm())
    assert all(c <= 1.1 * w for c, w in zip(off["chunks"], off["walk"])), off


@pytest.mark.parametrize("decays", ["channel", "head", "steep"])
@pytest.mark.parametrize("what", ["v", "k", "q"])
def test_what_a_token_brings_does_not_reach_the_tokens_before_it(decays, what, monkeypatch):
    """An infinity or a NaN in one token's row: every token before it keeps its output to the bit, wherever in a chunk it
    lies (in the chunks' products a later key has the weight 0, and 0 times an infinity is NaN)."""
    o, n, heads, d = ops(), 130, 2, 48
    monkeypatch.setattr(o, "GLA_LONG", 0)
    rows = {x: rnd(n, heads * d, seed=70 + i).bfloat16() for i, x in enumerate("qkv")}
    z = None if decays == "head" else rnd(n, heads * d, seed=73) * 3 - 2 if decays == "steep" else rnd(n, heads * d, seed=73) + 1
    hd = torch.tensor([0.9, 0.99]).to(DEV) if decays == "head" else None

    def run(rows):
        state = torch.zeros(1, heads, d, d, device=DEV)
        return o.gla_scan(*(rows[x].to(DEV) for x in "qkv"), None if z is None else z.to(DEV), None, 1.0, 1.0, heads, d, d, state,
                          ctx_for([n], [0]), head_decay=hd).cpu()
    clean = run(rows)
    assert torch.isfinite(clean).all()
    for at, bad in ((1, math.inf), (2, math.nan), (3, math.inf), (19, -math.inf), (34, math.nan), (63, math.inf), (66, math.inf), (129, math.nan)):
        spoilt = dict(rows)
        spoilt[what] = rows[what].clone()
        spoilt[what][at] = bad
        assert torch.equal(run(spoilt)[:at], clean[:at]), at


@pytest.mark.parametrize("decays", ["channel", "head", "token"])
@pytest.mark.parametrize("at", [0, 31, 40, 63, 64, 100, 129])
def test_an_infinite_key_leaves_what_it_leaves_in_the_walk(decays, at, monkeypatch):
    """One channel of one key is infinite: that row of the state becomes infinite with the values' signs, the outputs from that
    token on with the query's too, and nothing becomes NaN; the rest is finite.  Chunks and walk agree in each."""
    o, n, heads, d = ops(), 130, 2, 48
    q, k, v = (rnd(n, heads * d, seed=70 + i).bfloat16() for i in range(3))
    k[at, 5], k[at, d + 7] = math.inf, -math.inf
    z = (rnd(n, heads * d, seed=73) + 4).to(DEV) if decays == "channel" else None
    hd = torch.tensor([0.9, 0.99]).to(DEV) if decays == "head" else None
    tg = torch.sigmoid(rnd(n, heads, 3, seed=74) + 4).to(DEV) if decays == "token" else None
    got = {}
    for form, limit in (("walk", n), ("chunks", 0)):
        monkeypatch.setattr(o, "GLA_LONG", limit)
        state = torch.zeros(1, heads, d, d, device=DEV)
        out = o.gla_scan(q.to(DEV), k.to(DEV), v.to(DEV), z, None, 1.0, 1.0, heads, d, d, state, ctx_for([n], [0]), head_decay=hd,
                         tok_gates=tg)
        got[form] = out.cpu(), state.cpu()
    for walk, chunks in zip(*got.values()):
        assert walk.isinf().any() and not walk.isnan().any() and not chunks.isnan().any()
        assert torch.equal(walk.isinf(), chunks.isinf()) and torch.equal(walk[walk.isinf()], chunks[walk.isinf()])


@pytest.mark.parametrize("scale", [1e15, 1e-15])
@pytest.mark.parametrize("fall", [20.0, 40.0, 60.0, 75.0])
def test_large_and_small_keys_beside_strong_decays(scale, fall, monkeypatch):
    """Keys and queries far from 1, decays that fall by e^-fall within a chunk: k / D and q D stay inside fp32 in every form that a
    chunk may take.  Against the token loop in float64, 200 roundings of the largest terms."""
    o, n, d = ops(), 100, 16
    monkeypatch.setattr(o, "GLA_LONG", 0)
    q, k, v = rnd(n, d, seed=70).bfloat16() / scale, rnd(n, d, seed=71).bfloat16() * scale, rnd(n, d, seed=72).bfloat16()
    z = torch.full((n, d), -math.log(math.expm1(fall / 64)))          # sigmoid(z) = e^(-fall / 64)
    alpha, S, size = torch.sigmoid(z.double()), torch.zeros(d, d, dtype=torch.float64), torch.zeros(d, d, dtype=torch.float64)
    state = torch.zeros(1, 1, d, d, device=DEV)
    got = o.gla_scan(q.to(DEV), k.to(DEV), v.to(DEV), z.to(DEV), None, 1.0, 1.0, 1, d, d, state, ctx_for([n], [0])).cpu().double()
    for t in range(n):
        add = k[t].double()[:, None] * v[t].double()[None, :]
        S, size = alpha[t][:, None] * S + add, alpha[t][:, None] * size + add.abs()
        assert ((got[t] - q[t].double() @ S).abs() <= 200 * 2.0 ** -24 * (q[t].double().abs() @ size)).all(), t


def test_steep_decays_in_chunks_take_no_longer_than_the_walk(monkeypatch):
    """Channels that all but die within a chunk go pair by pair (743 us where the walk takes 1026; the gates evaluated anew
    for every pair took 2635): 1.5 times the walk's time is the bound, for the noise of a timer."""
    o, n, heads, d = ops(), 2000, 32, 128
    q, k, v = (rnd(n, heads * d, seed=i).bfloat16().to(DEV) for i in (70, 71, 72))
    z, state, ctx = (rnd(n, heads * d, seed=73) * 3 - 2).to(DEV), torch.zeros(1, heads, d, d, device=DEV), ctx_for([n], [0])

    def time(limit):
        monkeypatch.setattr(o, "GLA_LONG", limit)
        best = math.inf
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            o.gla_scan(q, k, v, z, None, 1.0, 1.0, heads, d, d, state, ctx)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best
    assert time(0) <= 1.5 * time(n)


@pytest.mark.parametrize("lens", [[1, 200, 33, 1, 64, 129, 5], [65, 64, 63], [1] * 300 + [150] + [2] * 20 + [64, 70]])
@pytest.mark.parametrize("longer_than", [None, 32])
@pytest.mark.parametrize("decays", ["channel", "head", "token"])
def test_linear_attention_of_unequal_portions_in_one_step(lens, longer_than, decays, monkeypatch):
    """Portions of every length in one call, against the token loop in float64 with the bound of the test above; a portion's
    numbers are to the bit those it gets alone, whatever shares the step; and scratch is taken for the chunks there are."""
    o, heads, dk, dv = ops(), 2, 48, 40
    if longer_than is not None:
        monkeypatch.setattr(o, "GLA_LONG", longer_than)
    Tn, starts = sum(lens), np.concatenate([[0], np.cumsum(lens)])
    q, k, v = rnd(Tn, heads * dk, seed=70).bfloat16(), rnd(Tn, heads * dk, seed=71).bfloat16(), rnd(Tn, heads * dv, seed=72).bfloat16()
    z = rnd(Tn, heads * dk, seed=73, scale=2.0) if decays == "channel" else None
    hd = torch.tensor([0.97, 0.6]) if decays == "head" else None
    tg = torch.sigmoid(rnd(Tn, heads, 3, seed=74) + 1) if decays == "token" else None
    S0 = rnd(len(lens), heads, dk, dv, seed=75)
    dev = lambda x, a, b: None if x is None else x[a:b].contiguous().to(DEV)

    def run(which):
        a, b = starts[which[0]], starts[which[-1] + 1]
        state = S0[which].to(DEV)
        out = o.gla_scan(dev(q, a, b), dev(k, a, b), dev(v, a, b), dev(z, a, b), None, 1.0, 1.0, heads, dk, dv, state,
                         ctx_for([lens[i] for i in which], list(range(len(which)))),
                         head_decay=None if hd is None else hd.to(DEV), tok_gates=dev(tg, a, b))
        return out.cpu(), state.cpu()

    run(list(range(len(lens))))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got, state = run(list(range(len(lens))))
    held = Tn * heads * (2 * dk + 2 * dv + 3 * dk + dv) * 4 + S0.numel() * 4
    chunks = sum(-(-n // 64) for n in lens)
    assert torch.cuda.max_memory_allocated() - before <= held + chunks * heads * (dk + dk * dv) * 4 + (1 << 21)
    alpha = (torch.sigmoid(z.double()).reshape(Tn, heads, dk) if z is not None else
             hd.double()[None, :, None].expand(Tn, heads, dk) if hd is not None else tg[..., :1].double().expand(Tn, heads, dk))
    kk = k.double().reshape(Tn, heads, dk) * (tg[..., 1:2].double() if tg is not None else 1.0)
    qq, vv = q.double().reshape(Tn, heads, dk), v.double().reshape(Tn, heads, dv)
    for i, n in enumerate(lens):
        S, size = S0[i].double(), S0[i].double().abs()
        rounds = 64 + (dk + 64) + 4 * (n // 64 + 1)
        for t in range(starts[i], starts[i] + n):
            add = kk[t][:, :, None] * vv[t][:, None, :]
            S, size = alpha[t][:, :, None] * S + add, alpha[t][:, :, None] * size + add.abs()
            want, terms = torch.einsum("hkv,hk->hv", S, qq[t]), torch.einsum("hkv,hk->hv", size, qq[t].abs())
            assert ((got[t].reshape(heads, dv).double() - want).abs() <= rounds * 2.0 ** -24 * terms + 1e-30).all(), (i, t)
        assert ((state[i].double() - S).abs() <= rounds * 2.0 ** -24 * size + 1e-30).all(), i
    for i in sorted({lens.index(n) for n in set(lens)}):
        alone, alone_state = run([i])
        assert torch.equal(alone, got[starts[i]:starts[i + 1]]) and torch.equal(alone_state[0], state[i]), i


@pytest.mark.parametrize("C,bw,taps,act,portions", [(48, 16, 4, "silu", (1, 2, 40, 33)), (40, 20, 3, None, (259,)), (24, 24, 2, None, (33, 256, 1)),
                                                    (36, 12, 4, None, (600,)), (40, 8, 5, "silu", (40, 1))])
def test_convolution_and_recurrent_unit_in_long_portions(C, bw, taps, act, portions):
    """The convolution on whole 16-byte pieces (C a multiple of 8, two to four taps) and element by element, and the
    unit's walk with 32 threads per channel at the edges of its rounds of 256 tokens, in bfloat16 against the plain
    formulas in float64 on the same rounded inputs: results are off by their rounding to bfloat16, 2^-8 of themselves, and the
    fp32 sums (the unit's state by 2^-20 of the largest)."""
    Tn = sum(portions)
    x, y = rnd(Tn, C, seed=80).bfloat16(), rnd(Tn, C, seed=81).bfloat16()
    w, b, xb, lam, yb = rnd(C, taps, seed=82), rnd(C, seed=83), rnd(C, seed=84), rnd(C, seed=85), rnd(C, seed=86)
    br, bi = rnd(C, seed=87), rnd(C, seed=88)
    gates = rnd(C // bw, Tn, 2 * bw, seed=89)
    state = torch.zeros(2, taps, C, device=DEV)
    us, outs, t0 = [], [], 0
    for n in portions:
        ctx, xs = ctx_for([n], [1]), x[t0:t0 + n].to(DEV)
        u = torch.empty(n, C, dtype=torch.bfloat16, device=DEV)
        ops().causal_conv(xs, xb.to(DEV), w.to(DEV), b.to(DEV), state, ctx, u, act=act)
        out = torch.empty(n, C, dtype=torch.bfloat16, device=DEV)
        ops().rglru_scan(gates[:, t0:t0 + n].contiguous().to(DEV), br.to(DEV), bi.to(DEV), lam.to(DEV), 8.0, u,
                         y[t0:t0 + n].to(DEV), yb.to(DEV), xs, xb.to(DEV), taps, state, ctx, out)
        us.append(u.cpu().double())
        outs.append(out.cpu().double())
        t0 += n
    u, out = torch.cat(us), torch.cat(outs)
    want = P.causal_conv(x.double() + xb.double(), w.double(), b.double())
    want = torch.nn.functional.silu(want) if act else want
    assert ((u - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
    r = torch.sigmoid(torch.cat(list(gates[:, :, :bw].double()), dim=1) + br.double())
    i = torch.sigmoid(torch.cat(list(gates[:, :, bw:].double()), dim=1) + bi.double())
    log_a = -8.0 * r * torch.nn.functional.softplus(lam.double())
    a, inp = log_a.exp(), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
    S, states = torch.zeros(C, dtype=torch.float64), []
    for t in range(Tn):
        S = a[t] * S + inp[t]
        states.append(S)
    ref = torch.stack(states) * P.gelu_tanh(y.double() + yb.double())
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()
    assert ((state[1, taps - 1].cpu().double() - S).abs() <= 2.0 ** -20 * torch.stack(states).abs().max()).all()
    assert torch.equal(state[1, :taps - 1].cpu(), (x.float() + xb)[Tn - (taps - 1):])


def unit_inputs(lens, C, bw, seed=80):
    n = sum(lens)
    g = {"gates": rnd(C // bw, n, 2 * bw, seed=seed)}
    g.update({k: rnd(n, C, seed=seed + i).bfloat16() for i, k in enumerate(("u", "y", "x"), 1)})
    g.update({k: rnd(C, seed=seed + i) * 0.1 for i, k in enumerate(("br", "bi", "lam", "yb", "xb"), 5)})
    return g


def run_unit(g, lens, which, S0, taps):
    starts = np.concatenate([[0], np.cumsum(lens)])
    a, b = starts[which[0]], starts[which[-1] + 1]
    d = {k: (v[:, a:b] if k == "gates" else v[a:b] if v.dim() == 2 else v).contiguous().to(DEV) for k, v in g.items()}
    state, out = S0[which].to(DEV), torch.empty(b - a, S0.shape[2], dtype=torch.bfloat16, device=DEV)
    ops().rglru_scan(d["gates"], d["br"], d["bi"], d["lam"], 8.0, d["u"], d["y"], d["yb"], d["x"], d["xb"], taps, state,
                     ctx_for([lens[i] for i in which], list(range(len(which)))), out)
    return out.cpu(), state.cpu()


@pytest.mark.parametrize("lens", [[1, 200, 33, 1, 64, 129, 5], [1] * 40 + [300] + [2] * 5])
@pytest.mark.parametrize("longer_than", [None, 32])
def test_recurrent_unit_of_unequal_portions_in_one_step(lens, longer_than, monkeypatch):
    """A portion's numbers are to the bit those it gets alone, whatever shares the step."""
    if longer_than is not None:
        monkeypatch.setattr(ops(), "RGLRU_LONG", longer_than)
    C, bw, taps = 40, 20, 4
    g, S0 = unit_inputs(lens, C, bw), rnd(len(lens), taps, C, seed=95)
    out, state = run_unit(g, lens, list(range(len(lens))), S0, taps)
    starts = np.concatenate([[0], np.cumsum(lens)])
    for i in sorted({lens.index(n) for n in set(lens)}):
        alone, alone_state = run_unit(g, lens, [i], S0, taps)
        assert torch.equal(alone, out[starts[i]:starts[i + 1]]) and torch.equal(alone_state[0], state[i]), i


@pytest.mark.parametrize("n", [65, 256, 300, 1000])
def test_recurrent_unit_of_long_portions_is_no_further_from_64_bits_than_the_walk(n, monkeypatch):
    """The state behind the portion, walked token by token in fp32 and by folds and a scan, both against float64."""
    C, bw, taps = 640, 64, 4
    g, S0 = unit_inputs([n], C, bw), rnd(1, taps, C, seed=95)
    r = torch.sigmoid(torch.cat(list(g["gates"][:, :, :bw].double()), dim=1) + g["br"].double())
    i = torch.sigmoid(torch.cat(list(g["gates"][:, :, bw:].double()), dim=1) + g["bi"].double())
    log_a = -8.0 * r * torch.nn.functional.softplus(g["lam"].double() - 3)
    a, inp = log_a.exp(), torch.sqrt(-torch.expm1(2 * log_a)) * i * g["u"].double()
    S = S0[0, taps - 1].double()
    for t in range(n):
        S = a[t] * S + inp[t]
    g["lam"] = g["lam"] - 3
    off = {}
    for form, limit in (("walk", n), ("scan", 0)):
        monkeypatch.setattr(ops(), "RGLRU_LONG", limit)
        off[form] = float((run_unit(g, [n], [0], S0, taps)[1][0, taps - 1].double() - S).norm())
    assert off["scan"] <= 1.02 * off["walk"], off


@pytest.mark.parametrize("K", [64, 256, 520, 1024, 2816, 8192])
def test_experts_of_few_rows_sum_as_fp32_would(K):
    """The fp32 result of the streaming product of few rows against float64.  Summing K products one by one in fp32 is off
    by about 2^-25 of the running sums, sqrt(K / 2) of a typical result: 32 chains of K / 32 fused multiply-adds and a tree over
    them, the order that an fp32 product of this kind has, are imitated here, and the kernel may be off by no more (an
    accumulator of tensor-core instructions carried through all of k is off by 1.4 times that at K = 512 and 4 at 2816; at K = 64
    even one instruction's sum of 16 is, and the CUDA cores take it)."""
    E, rows, H = 3, 8, 128
    a = rnd(E * rows, K, seed=90).bfloat16()
    w = rnd(E, H, K, seed=91, scale=K ** -0.5).bfloat16()
    plan = torch.tensor([E] + [rows * e for e in range(E + 1)] + [x for e in range(E) for x in (e, rows * e, rows)]
                        + [0] * (3 * E), dtype=torch.int32, device=DEV)
    y = torch.empty(E * rows, H, device=DEV)
    ad, wd = a.to(DEV), w.to(DEV)
    lib = ops()._lib("moe")
    rc = lib.mi_moe_down(ad.data_ptr(), wd.data_ptr(), H * K, plan.data_ptr(), E, y.data_ptr(), E * rows, H, K, 8, 0, 1,
                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    prod = (a.double().reshape(E, rows, 1, K) * w.double().reshape(E, 1, H, K)).reshape(E * rows, H, K)
    want = prod.sum(dim=-1)
    pad = -K % 256
    lanes = torch.nn.functional.pad(prod, (0, pad)).reshape(E * rows, H, -1, 32, 8).permute(0, 1, 3, 2, 4).flatten(3)
    acc = torch.zeros(E * rows, H, 32)
    for i in range(lanes.shape[-1]):            # a product of two bfloat16 is exact, so this rounds as a fused multiply-add
        acc = (acc.double() + lanes[..., i]).float()
    while acc.shape[-1] > 1:
        acc = acc[..., :acc.shape[-1] // 2] + acc[..., acc.shape[-1] // 2:]
    fp32 = (acc[..., 0].double() - want).norm()
    assert (y.cpu().double() - want).norm() <= fp32


@pytest.mark.parametrize("E,top,ff,H,M", [(5, 2, 24, 40, 33), (3, 1, 20, 48, 5), (4, 4, 16, 36, 70), (12, 3, 72, 64, 200),
                                          (6, 2, 24, 40, 7), (3, 3, 16, 64, 8), (16, 1, 8, 264, 100)])
@pytest.mark.parametrize("dtype,bound", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2)])
def test_routed_experts(E, top, ff, H, M, dtype, bound):
    """Router choice and weights, the clamped activation, and the weighted sum, against the plain
    token loop; the inputs are scaled so that both clamps bite."""
    x = rnd(M, H, seed=60).to(dtype)
    W = {"router": rnd(E, H, seed=61, scale=0.5).to(dtype)}
    for e in range(E):
        W[f"e{e}.gate"] = rnd(ff, H, seed=100 + e, scale=0.4).to(dtype)
        W[f"e{e}.up"] = rnd(ff, H, seed=200 + e, scale=0.4).to(dtype)
        W[f"e{e}.down"] = rnd(H, ff, seed=300 + e, scale=0.2).to(dtype)
    mlp = {"router": {"experts": E, "top": top}, "expert": {"ff": ff, "limit": 0.9}}
    margins = []
    want = P.moe(x.double(), {k: v.double() for k, v in W.items()}, mlp, margins)
    dx = x.to(DEV)
    ids, wts = ops().moe_route(dx, W["router"].to(DEV), top)
    z = x.double() @ W["router"].double().T
    ok = torch.ones(M, dtype=torch.bool) if not margins else margins[0] > 1e-3
    vals, idx = torch.topk(z, top, dim=-1)
    assert torch.equal(ids.cpu().long()[ok], idx[ok])
    assert (wts.cpu().double()[ok] - torch.softmax(vals, dim=-1)[ok]).abs().max() < 1e-5
    gate_up = torch.stack([torch.cat([W[f"e{e}.gate"], W[f"e{e}.up"]]) for e in range(E)]).to(DEV).contiguous()
    down = torch.stack([W[f"e{e}.down"] for e in range(E)]).to(DEV).contiguous()
    shared = rnd(M, H, seed=62).to(dtype)
    out = ops().moe_experts(dx, ids, wts, gate_up, down, 0.9, 1.702, shared.to(DEV))
    ref = want + shared.double()
    assert (out.cpu().double() - ref)[ok].abs().max() <= bound * max(1.0, ref.abs().max())


def test_window_edges_page_borders_and_far_keys():
    """One key is made to stand out (its direction is the queries', ten times longer in value): a
    query whose window still holds it returns its value, the next one does not; the key sits at a
    page's last slot, at a page's first slot, and hundreds of tokens back with no window at all."""
    from mini_infer_b200.engine import ModelRunner, StepEntry
    from mini_infer_b200.parts.base import LayerCache

    def run(window, n_tokens, marked, page):
        nq, nkv, d, dv = 2, 1, 16, 12
        cfg = {"architecture": "Ruvurax", "vocab": 8, "width": 16, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6},
               "layers": [{"type": "parallel", "mlp": None,
                           "mixer": {"left": {"heads": nq, "kv_heads": nkv, "dim": d, "vdim": dv,
                                              "mask": {"size": window} if window else None,
                                              "rot": None, "scale": 4.0},
                                     "right": {"heads": 1, "dim": 4, "vdim": 4, "tau": 2.0},
                                     "left_scale": 1.0, "right_scale": 1.0}}]}
        state = random_state(cfg, seed=3, rank=2)
        runner = ModelRunner.from_state_dict(cfg, state, dtype="float32", block_size=page,
                                             num_blocks=-(-n_tokens // page) + 1, max_requests=2)
        for st in runner.cache.storage:
            st.fill_(float("nan"))
        runner.add_request("a")
        ctx, caches, _, _ = runner.stepper.plan([StepEntry("a", [0] * n_tokens, [])])
        runner.stepper.apply_table_updates(ctx)
        cache = caches[0]
        # packed q | k | v: every query and key points along e0; the marked key is as long as the others
        # (unit norm equalises them anyway) but all other keys point along e1, so only it scores high
        packed = torch.zeros(n_tokens, (nq + nkv) * d + nkv * dv)
        packed[:, 0:nq * d:d] = 1.0                          # q heads: e0
        packed[:, nq * d + 1] = 1.0                          # keys: e1
        packed[marked, nq * d + 1] = 0.0
        packed[marked, nq * d] = 1.0                         # the marked key: e0
        packed[:, (nq + nkv) * d:] = 1.0                     # values: ones ...
        packed[marked, (nq + nkv) * d:] = 10.0               # ... the marked value: tens
        dev = packed.to(DEV)
        ops().rope_norm_store(dev, 0, nq * d, (nq + nkv) * d, nq, nkv, d, dv, positions=None, inv_freq=None, rot=0,
                              unit_norm=True, eps=1e-6, slots=ctx.groups[cache.group].slots, kcache=cache.k,
                              vcache=cache.v)
        out = torch.empty(n_tokens, nq * dv, device=DEV)
        ops().attention_kv(dev[:, :nq * d], out, cache, ctx, nq, nkv, d, dv, 4.0, window or 0)
        return out.cpu()

    # score of the marked key: q.k * scale = 16 * 4 = 64 above the others: its weight is 1 to fp32 precision
    for page, marked in ((8, 15), (8, 16), (16, 31), (4, 13)):       # last slot of a page, first slot, inside
        window = 11
        out = run(window, 64, marked, page)
        for i in range(64):
            sees = 0 <= i - marked < window
            assert torch.allclose(out[i], torch.full_like(out[i], 10.0 if sees else 1.0), atol=1e-4), (page, marked, i)
    out = run(None, 700, 3, 16)                                      # no window: a key 696 tokens back
    assert torch.allclose(out[3:], torch.full_like(out[3:], 10.0), atol=1e-4)
    assert torch.allclose(out[:3], torch.full_like(out[:3], 1.0), atol=1e-4)

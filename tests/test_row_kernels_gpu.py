"""The forms of the small row kernels that take whole aligned pieces against those that take any row: the same call on a
tensor that starts four bytes off, or with a width that is no multiple of a piece, reaches the other form."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def ops():
    from mini_infer_b200.csrc import ops as o
    return o


def rnd(*shape, dtype=torch.float32, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(DEV)


def shifted(t):
    """The same numbers at an address that is no multiple of 16."""
    flat = torch.empty(t.numel() + 2, dtype=t.dtype, device=t.device)[2:]
    flat.copy_(t.reshape(-1))
    return flat.view(t.shape)


def bound(dtype, want):
    # a norm of fp32 sums over up to 8192 numbers in two orders: some ulps; a bfloat16 result may round the other way
    return (2.0 ** -7 if dtype == torch.bfloat16 else 1e-5) * want.abs().max().clamp(min=1.0).item()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,H", [(1, 4), (3, 516), (8, 2048), (5, 2052), (2, 4096), (3, 8192), (2, 8196), (4, 4099)])
def test_layer_norm_in_registers(dtype, M, H):
    o = ops()
    stream, a1, a2 = rnd(M, H, seed=1), rnd(M, H, dtype=dtype, seed=2), rnd(M, H, dtype=dtype, seed=3)
    w1, b1, w2, b2 = (rnd(H, seed=s) for s in (4, 5, 6, 7))
    r = stream.double() + a1.double() + a2.double()
    n = (r - r.mean(dim=1, keepdim=True)) * torch.rsqrt(r.var(dim=1, unbiased=False, keepdim=True) + 1e-6)
    for adds in ((a1, a2), (shifted(a1), a2)):
        new = stream.clone()
        out1, out2 = o.add_layernorm(new, adds, [(w1, b1), (w2, b2)], 1e-6, dtype)
        assert (new.double() - r).abs().max().item() <= 1e-6 * r.abs().max().item()
        for got, w, b in ((out1, w1, b1), (out2, w2, b2)):
            want = n * w.double() + b.double()
            assert (got.double() - want).abs().max().item() <= bound(dtype, want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,H", [(1, 8), (3, 516), (8, 2048), (2, 4096), (3, 8192), (2, 8196), (4, 4099)])
def test_norm_of_several_addends_in_registers(dtype, M, H):
    o = ops()
    stream, add32, row_add, gain = rnd(M, H, seed=1), rnd(M, H, seed=2), rnd(H, seed=3), rnd(H, seed=4)
    a1, a2 = rnd(M, H, dtype=dtype, seed=5), rnd(M, H, dtype=dtype, seed=6)
    for adds, extra in (((a1, a2), True), ((shifted(a1), a2), True), ((a1,), False), ((), True)):
        kw = dict(add32=add32, row_add=row_add) if extra else {}
        r = stream.double() + sum(a.double() for a in adds) + ((add32.double() + row_add.double()) if extra else 0.0)
        want = gain.double() * r * torch.rsqrt((r * r).mean(dim=1, keepdim=True) + 1e-6)
        out, new = o.add_rmsnorm_multi(stream, adds, gain, 1e-6, dtype, **kw)
        assert (new.double() - r).abs().max().item() <= 1e-6 * r.abs().max().item()
        assert (out.double() - want).abs().max().item() <= bound(dtype, want)
        with o.kept_sums():                   # the order that kept sums have: close, and the same stream
            kept, stream_kept = o.add_rmsnorm_multi(stream, adds, gain, 1e-6, dtype, **kw)
        assert torch.equal(stream_kept, new) and (kept.double() - want).abs().max().item() <= bound(dtype, want)


@pytest.mark.parametrize("act", ["sigmoid", "silu"])
@pytest.mark.parametrize("M,C,per", [(1, 8, 1), (3, 264, 1), (70, 1024, 1), (5, 256, 128), (5, 96, 8), (4, 96, 4), (3, 100, 1)])
def test_gate_in_pieces_has_the_bits_of_single_elements(M, C, per, act):
    o = ops()
    x, g = rnd(M, C + 24, dtype=torch.bfloat16, seed=1)[:, 8:8 + C], rnd(M, C // per, dtype=torch.bfloat16, seed=2)
    out, single = (torch.empty(M, C, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    o.gate_mul(x, g, out, act, 0.5, per=per)
    o.gate_mul(shifted(x.contiguous()), g, single, act, 0.5, per=per)
    assert torch.equal(out, single)
    z = g.double().repeat_interleave(per, dim=1)
    want = x.double() * torch.sigmoid(z) * (z if act == "silu" else 1.0) * 0.5
    assert (out.double() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M", [3, 70])
@pytest.mark.parametrize("d,rot", [(64, 64), (64, 0), (128, 128), (128, 64), (128, 0), (256, 256), (256, 128), (128, 32), (96, 96)])
def test_normed_and_rotated_heads_in_registers(dtype, M, d, rot):
    """Heads whose pairs lie in one lane, and (the last two) those that go through shared memory, against float64."""
    o, nq, nkv, page = ops(), 5, 2, 8
    x = rnd(M, (nq + 2 * nkv) * d, dtype=dtype, seed=1)
    qg, kg = rnd(d, seed=2), rnd(d, seed=3)
    positions = torch.arange(M, dtype=torch.int32, device=DEV) * 37 + 5
    freq = 10000.0 ** (-torch.arange(0, max(rot, 2), 2, dtype=torch.float64, device=DEV) / max(rot, 2))
    caches = [torch.zeros(-(-M // page), nkv, page, d, dtype=dtype, device=DEV) for _ in range(2)]
    packed = x.clone()
    o.qk_norm_rope_store(packed, 0, nq * d, (nq + nkv) * d, nq, nkv, d, d, q_gain=qg, k_gain=kg, eps=1e-6, rot=rot,
                         positions=positions, freq=freq if rot else None, slots=torch.arange(M, dtype=torch.int32, device=DEV),
                         kcache=caches[0], vcache=caches[1])
    heads = x.double().view(M, -1, d)
    for first, n, gain in ((0, nq, qg), (nq, nkv, kg)):
        h = heads[:, first:first + n]
        y = h * torch.rsqrt((h * h).mean(dim=-1, keepdim=True) + 1e-6) * gain.double()
        if rot:
            ang = positions.double()[:, None, None] * freq
            u, v = y[..., :rot // 2].clone(), y[..., rot // 2:rot].clone()
            y[..., :rot // 2], y[..., rot // 2:rot] = u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()
        got = packed.double().view(M, -1, d)[:, first:first + n]
        assert (got - y).abs().max().item() <= bound(dtype, y)
    rows = o.unpack_cache_pages(caches[0])[:M].reshape(M, -1)
    assert torch.equal(rows, packed[:, nq * d:(nq + nkv) * d])
    assert torch.equal(o.unpack_cache_pages(caches[1])[:M].reshape(M, -1), x[:, (nq + nkv) * d:])


def cache_pair(M, nkv, d, page, dtype):
    return [torch.zeros(-(-M // page), nkv, page, d, dtype=dtype, device=DEV) for _ in range(2)]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M", [2, 70])
@pytest.mark.parametrize("nq,nkv,d,rot", [(3, 1, 2, 2), (32, 8, 128, 64), (5, 2, 100, 10), (2, 1, 256, 256)])
def test_rotated_unit_heads_in_pairs_have_the_bits_of_single_elements(dtype, M, nq, nkv, d, rot):
    o, page = ops(), 8
    width = (nq + 2 * nkv) * d
    x = rnd(M, width, dtype=dtype, seed=1)
    inv = 1000.0 ** (-torch.arange(0, rot, 2, dtype=torch.float32, device=DEV) / rot)
    slots = torch.arange(M, dtype=torch.int32, device=DEV)
    results = []
    for off in (0, 1):               # from the second column on a pair is no aligned access
        wide = torch.zeros(M, width + 2, dtype=dtype, device=DEV)
        packed = wide[:, off:off + width]
        packed.copy_(x)
        k, v = cache_pair(M, nkv, d, page, dtype)
        o.rope_norm_store(packed, 0, nq * d, (nq + nkv) * d, nq, nkv, d, d, positions=slots * 37 + 5, inv_freq=inv, rot=rot,
                          unit_norm=True, eps=1e-6, slots=slots, kcache=k, vcache=v)
        results.append((packed.clone(), k, v))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    h = x.double().view(M, -1, d)[:, :nq + nkv]
    ang = (slots * 37 + 5).float()[:, None, None] * inv
    y, u, w = h.clone(), h[..., 0:rot:2], h[..., 1:rot:2]
    y[..., 0:rot:2] = u * ang.double().cos() - w * ang.double().sin()
    y[..., 1:rot:2] = w * ang.double().cos() + u * ang.double().sin()
    y = y * torch.rsqrt((y * y).mean(dim=-1, keepdim=True) + 1e-6)
    assert (results[0][0].double().view(M, -1, d)[:, :nq + nkv] - y).abs().max().item() <= bound(dtype, y)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M", [2, 70])
@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("d", [4, 64, 128, 132, 256])
def test_biased_and_normed_heads_in_pieces(dtype, M, own, d):
    o, nq, nkv, page = ops(), 6, 2, 8
    width = (nq + (2 if own else 1) * nkv) * d
    x, slots = rnd(M, width, dtype=dtype, seed=1), torch.arange(M, dtype=torch.int32, device=DEV)
    qb, kb, qg, kg = rnd(nq * d, seed=2), rnd(nkv * d, seed=3), rnd(d, seed=4), rnd(d, seed=5)
    h = x.double().view(M, -1, d)[:, :nq + nkv] + torch.cat([qb, kb]).double().view(-1, d)
    want = h * torch.rsqrt((h * h).mean(dim=-1, keepdim=True) + 1e-6)
    want = want * torch.cat([qg.expand(nq, d), kg.expand(nkv, d)]).double()
    for off in (0, 1):
        wide = torch.zeros(M, width + 4, dtype=dtype, device=DEV)
        packed = wide[:, off:off + width]
        packed.copy_(x)
        k, v = cache_pair(M, nkv, d, page, dtype)
        o.qk_bias_norm_store(packed, 0, nq * d, (nq + nkv) * d if own else nq * d, nq, nkv, d, d, q_bias=qb, k_bias=kb, q_gain=qg,
                             k_gain=kg, eps=1e-6, values_are_keys=not own, slots=slots, kcache=k, vcache=v)
        got = packed.double().reshape(M, -1, d)[:, :nq + nkv]
        assert (got - want).abs().max().item() <= bound(dtype, want)
        assert torch.equal(o.unpack_cache_pages(k)[:M].reshape(M, -1), packed[:, nq * d:(nq + nkv) * d])
        values = o.unpack_cache_pages(v)[:M]
        if own:
            assert torch.equal(values.reshape(M, -1), x[:, (nq + nkv) * d:])
        else:
            assert (values.double() - h[:, nq:]).abs().max().item() <= bound(dtype, h)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kvh,dk,dv", [(2, 1, 20, 33), (3, 3, 32, 8), (4, 2, 64, 64), (2, 2, 100, 37), (1, 1, 128, 40),
                                             (2, 1, 128, 128)])
@pytest.mark.parametrize("lens", [(33, 41), (32, 15), (34, 1), (130, 8), (16, 56)])
def test_delta_rule_with_warps_that_stage(dtype, heads, kvh, dk, dv, lens):
    """A long portion, staged by warps of its own, against the same tokens in portions too short for that: one order of
    sums, so the outputs, the states and the convolution's tails are equal bit by bit."""
    from types import SimpleNamespace
    gk, taps = kvh * dk, 3
    C = 2 * gk + heads * dv
    s_off = (taps - 1) * C
    n = sum(lens)
    u, x, z = rnd(n, C, dtype=dtype, seed=1), rnd(n, C, dtype=dtype, seed=2), rnd(n, heads * dk, seed=3)
    b, dt, a_log = rnd(n, heads, dtype=dtype, seed=4), rnd(heads * dk, seed=5), rnd(heads, seed=6) - 0.5
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)

    def scan(starts, portions, slots, state):
        ctx = SimpleNamespace(q_start=i32(*starts), q_len=i32(*portions), state_slot=i32(*slots), n_requests=len(portions),
                              decode_only=max(portions) == 1, host_q_len=list(portions))
        return ops().delta_scan(u[:, :gk], u[:, gk:2 * gk], u[:, 2 * gk:], z, dt, a_log, b, dk ** -0.5, 1e-6, heads, kvh,
                                dk, dv, state, s_off, ctx, conv_in=x, taps=taps)

    begin = rnd(3, s_off + heads * dk * dv, seed=7)
    whole, cut = begin.clone(), begin.clone()
    got = scan((0, lens[0]), lens, (2, 0), whole)
    want = torch.empty_like(got)
    for start, length, slot in ((0, lens[0], 2), (lens[0], lens[1], 0)):
        for t in range(0, length, 7):
            m = min(7, length - t)
            want[start + t:start + t + m] = scan((start + t,), (m,), (slot,), cut)[start + t:start + t + m]
    assert torch.isfinite(got).all()
    assert torch.equal(got, want) and torch.equal(whole, cut)
    assert torch.equal(whole[1], begin[1])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,H", [(1, 4), (3, 100), (3, 508), (3, 516), (2, 1028), (8, 2048), (5, 2052), (2, 4096), (2, 4100), (3, 8192)])
def test_norms_in_registers_have_the_bits_of_the_form_for_any_row(dtype, M, H):
    """One order of sums whatever the address, the kept sums of models with groups of experts among them."""
    o = ops()
    stream, a1, a2, add32 = rnd(M, H, seed=1), rnd(M, H, dtype=dtype, seed=2), rnd(M, H, dtype=dtype, seed=3), rnd(M, H, seed=8)
    w1, b1, w2, b2 = (rnd(H, seed=s) for s in (4, 5, 6, 7))
    rows = torch.tensor([M - 1, 0], dtype=torch.int32, device=DEV)
    for adds in ((a1, a2), (a1,), ()):
        got = []
        for w in (w1, shifted(w1)):           # a gain at any address takes the other form
            new = stream.clone()
            outs = o.add_layernorm(new, adds, [(w, b1), (w2, b2)], 1e-6, dtype)
            got.append([*outs, new, *o.add_layernorm(stream, adds, [(w, b1)], 1e-6, dtype, rows=rows)])
            for s, kw in ((stream, {}), (stream, dict(add32=add32, row_add=b1)), (None, dict(add32=add32))):
                got[-1] += o.add_rmsnorm_multi(s, adds, w, 1e-6, dtype, **kw)
            got[-1].append(o.add_rmsnorm_multi(stream, adds, w, 1e-6, dtype, rows=rows)[0])
        assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M", [2, 70])
@pytest.mark.parametrize("d", [4, 20, 64, 100, 128, 132, 252, 256])
def test_biased_heads_in_pieces_have_the_bits_of_single_elements(dtype, M, d):
    o, nq, nkv, page = ops(), 6, 2, 8
    width = (nq + nkv) * d
    x, slots = rnd(M, width, dtype=dtype, seed=1), torch.arange(M, dtype=torch.int32, device=DEV)
    qb, kb, qg, kg = rnd(nq * d, seed=2), rnd(nkv * d, seed=3), rnd(d, seed=4), rnd(d, seed=5)
    for bias in (True, False):
        got = []
        for off in (0, 1):               # from the second column on a piece is no aligned access
            packed = torch.zeros(M, width + 4, dtype=dtype, device=DEV)[:, off:off + width]
            packed.copy_(x)
            k, v = cache_pair(M, nkv, d, page, dtype)
            o.qk_bias_norm_store(packed, 0, nq * d, nq * d, nq, nkv, d, d, q_bias=qb if bias else None, k_bias=kb if bias else None,
                                 q_gain=qg, k_gain=kg, eps=1e-6, values_are_keys=True, slots=slots, kcache=k, vcache=v)
            got.append((packed, k, v))
        assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("dtype", DTYPES)
def test_gains_that_the_kernel_before_writes(dtype):
    """Gain and bias are results of a long product of this library right in front of the norm: unless the caller says that they are
    constant, no kernel may read them before that product is done."""
    o, M, H, K = ops(), 3, 2048, 8192
    x, w, stream, add = rnd(1, K, seed=1), rnd(H, K, seed=2), rnd(M, H, seed=3), rnd(M, H, dtype=dtype, seed=4)
    gain = torch.full((1, H), float("nan"), device=DEV)
    norms = [lambda g, **kw: o.add_layernorm(stream, [add], [(g, g)], 1e-6, dtype, update_stream=False, **kw)[0],
             lambda g, **kw: o.add_layernorm(stream, [add], [(g, g), (g, g)], 1e-6, dtype, update_stream=False, **kw)[1],
             lambda g, **kw: o.add_rmsnorm_multi(stream, [add], g, 1e-6, dtype, **kw)[0]]
    for norm in norms:
        for _ in range(5):
            gain.fill_(float("nan"))
            torch.cuda.synchronize()
            o.gemm_f32(x, w, out=gain)
            got = norm(gain[0])
            torch.cuda.synchronize()
            want = norm(gain[0].clone())
            assert torch.isfinite(want).all() and torch.equal(got, want)
        assert torch.equal(norm(gain[0], w_constant=True), want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("M,heads,dv", [(1, 2, 64), (3, 3, 128), (70, 2, 256), (5, 4, 96), (2, 2, 288)])
def test_gated_norm_of_heads_in_lanes_and_in_a_loop(dtype, per_head, M, heads, dv):
    """Heads of 64, 128 and 256 stay in registers, others (the last two) are walked: against float64, with one gain for all heads
    and one for each, without a gate and with either."""
    o = ops()
    x, g = rnd(M, heads * dv, seed=1), rnd(M, heads * dv, dtype=dtype, seed=2)
    w = rnd(heads * dv if per_head else dv, seed=3)
    h = x.double().view(M, heads, dv)
    y = h * torch.rsqrt((h * h).mean(dim=-1, keepdim=True) + 1e-6) * (w.double().view(heads, dv) if per_head else w.double())
    for act in (None, "sigmoid", "silu"):
        out = torch.empty(M, heads * dv, dtype=dtype, device=DEV)
        o.headnorm_gate(x, w, None if act is None else g, out, heads, dv, 1e-6, act, 0.7)
        z = g.double().view(M, heads, dv)
        want = 0.7 * y * (1.0 if act is None else torch.sigmoid(z) * (z if act == "silu" else 1.0))
        assert (out.double().view(M, heads, dv) - want).abs().max().item() <= bound(dtype, want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,H", [(1, 8), (31, 12), (32, 8), (33, 7), (65, 512)])
def test_pair_hash_embedding_of_many_requests(dtype, n, H):
    """A token's request is looked for 32 requests at a time; portions of 0 to 3 tokens."""
    from types import SimpleNamespace
    V, buckets, mul_prev, mul_cur = 50, 37, 7919, 104729
    lens = [(5 * i + 1) % 4 for i in range(n)]
    lens[0] = lens[-1] = 2
    starts = [sum(lens[:i]) for i in range(n)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    ids = [(11 * t + 3) % V for t in range(sum(lens))]
    before = [(3 * i + 1) % V for i in range(n)]
    first = [i % 3 == 0 for i in range(n)]              # sequences at their beginning
    positions = [(0 if f else 9) + j for f, m in zip(first, lens) for j in range(m)]
    table, pairs = rnd(V, H, dtype=dtype, seed=1), rnd(buckets + 1, H, dtype=dtype, seed=2)
    slots = [(7 * i) % n if n % 7 else i for i in range(n)]
    last = torch.zeros(n, 1, dtype=torch.int32, device=DEV)
    for i, s in enumerate(slots):
        last[s] = before[i]
    ctx = SimpleNamespace(token_ids=i32(ids), positions=i32(positions), q_start=i32(starts), q_len=i32(lens), state_slot=i32(slots),
                          n_requests=n, n_tokens=len(ids))
    out = ops().embedding_pair_hash(table, pairs, ctx, last, buckets, mul_prev, mul_cur)
    for i, (start, m) in enumerate(zip(starts, lens)):
        prev = None if first[i] else before[i]
        for t in range(start, start + m):
            row = buckets if prev is None else (prev * mul_prev + ids[t] * mul_cur) % buckets
            assert torch.equal(out[t], table[ids[t]].float() + pairs[row].float()), (i, t)
            prev = ids[t]
        if m:
            assert last[slots[i], 0].item() == ids[start + m - 1]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M", [1137, 1139, 2730, 2731])
def test_heads_of_many_tokens_have_the_bits_of_few(dtype, M):
    """A warp takes one, two or four heads by the number of tokens times heads (9 a token here: 10240 and 24576 lie between the
    sizes): what a token gives does not depend on it."""
    o, nq, nkv, d, page = ops(), 5, 2, 64, 16
    width, pages = (nq + 2 * nkv) * d, -(-M // page)
    x, slots = rnd(M, width, dtype=dtype, seed=1), torch.arange(M, dtype=torch.int32, device=DEV)
    inv = 1000.0 ** (-torch.arange(0, d, 2, dtype=torch.float32, device=DEV) / d)
    gains, bias = (rnd(d, seed=2), rnd(d, seed=3)), (rnd(nq * d, seed=4), rnd(nkv * d, seed=5))
    calls = [lambda p, s, k, v: o.rope_norm_store(p, 0, nq * d, (nq + nkv) * d, nq, nkv, d, d, positions=s * 3 + 1, inv_freq=inv,
                                                  rot=d, unit_norm=True, eps=1e-6, slots=s, kcache=k, vcache=v),
             lambda p, s, k, v: o.qk_norm_rope_store(p, 0, nq * d, (nq + nkv) * d, nq, nkv, d, d, q_gain=gains[0], k_gain=gains[1],
                                                     eps=1e-6, rot=d, positions=s * 3 + 1, freq=inv.double(), slots=s, kcache=k,
                                                     vcache=v),
             lambda p, s, k, v: o.qk_bias_norm_store(p, 0, nq * d, (nq + nkv) * d, nq, nkv, d, d, q_bias=bias[0], k_bias=bias[1],
                                                     q_gain=gains[0], k_gain=gains[1], eps=1e-6, values_are_keys=False, slots=s,
                                                     kcache=k, vcache=v)]
    for call in calls:
        whole, cut = (x.clone() for _ in range(2))
        caches = [cache_pair(pages * page, nkv, d, page, dtype) for _ in range(2)]
        call(whole, slots, *caches[0])
        for t in range(0, M, 100):
            call(cut[t:t + 100], slots[t:t + 100], *caches[1])
        assert torch.equal(whole, cut) and all(torch.equal(a, b) for a, b in zip(*caches))

"""Tokens whose router logits leave no expert to choose, and ids that are no expert's: every id and place stays in range, the
tokens concerned come out NaN, and the other tokens of the step have the bits that they have without them."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from mini_infer_b200.csrc import ops as o
    return o


def rnd(*shape, dtype=torch.float32, seed=0, scale=1.0):
    return (scale * torch.randn(*shape, generator=torch.Generator().manual_seed(seed))).to(dtype).to(DEV)


def select(logits, top, mode, groups=0, keep=0):
    o = ops()
    M, E = logits.shape
    ids = torch.empty(M, top, dtype=torch.int32, device=DEV)
    weights = torch.empty(M, top, device=DEV)
    lib = o._lib("moe")
    rc = lib.mi_moe_select(o._ptr(logits), E, o._ptr(ids), o._ptr(weights), M, E, top, o.ROUTE_MODES[mode], groups, keep, 1.5,
                           None, 0, None, o._stream())
    o._finish(lib, rc, "moe_select")
    return ids, weights


@pytest.mark.parametrize("mode", ["chosen", "all", "sigmoid"])
@pytest.mark.parametrize("E,top,groups", [(4, 4, 0), (32, 4, 4), (33, 5, 0), (64, 8, 8), (65, 8, 0), (256, 32, 8)])
def test_tokens_without_a_candidate_get_valid_ids_and_weights_that_show_it(E, top, groups, mode):
    good = rnd(5, E, seed=E)
    logits = torch.cat([good, torch.zeros(3, E, device=DEV)])
    logits[5], logits[6] = float("nan"), float("-inf")
    logits[7, 1:] = float("-inf") if mode != "sigmoid" else float("nan")      # one candidate (a sigmoid makes 0 of -inf: one too)
    keep = groups // 2
    ids, weights = select(logits, top, mode, groups, keep)
    assert int(ids.min()) >= 0 and int(ids.max()) < E
    want_ids, want = select(good, top, mode, groups, keep)
    assert torch.equal(ids[:5], want_ids) and torch.equal(weights[:5], want) and torch.isfinite(want).all()
    assert torch.isnan(weights[5]).any() and torch.isnan(weights[7]).any() and int(ids[7, 0]) == 0
    if mode != "sigmoid":
        assert torch.isnan(weights[6]).any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,E", [(9, 16), (9, 2), (200, 4)])      # few rows per expert, 64-row tiles, the library's grouped product
def test_ids_that_are_no_experts_leave_the_other_tokens_alone(M, E, dtype):
    o, H, ff, top = ops(), 64, 32, 2
    x, gate_up, down = (rnd(*s, dtype=dtype, seed=i, scale=0.3) for i, s in enumerate(((M, H), (E, 2 * ff, H), (E, H, ff))))
    ids = torch.stack([torch.arange(M) % E, (torch.arange(M) + 1) % E], dim=1).to(torch.int32).to(DEV)
    weights = rnd(M, top, seed=5)
    run = lambda i: o.moe_experts(x, i, weights, gate_up, down, float("inf"), 1.0, None, up_offset=0.0)
    bad = ids.clone()
    bad[1, 0], bad[3, 1], bad[4, 0], bad[M - 1, 1] = 0x7fffffff, -1, E, -0x7fffffff
    broken = [1, 3, 4, M - 1]
    rest = [t for t in range(M) if t not in broken]
    want, got = run(ids), run(bad)
    assert torch.isfinite(want).all() and torch.isnan(got[broken]).all()
    assert torch.equal(got[rest], want[rest])
    with o.kept_sums():
        want, got = run(ids), run(bad)
    assert torch.isnan(got[broken]).all() and torch.equal(got[rest], want[rest])


@pytest.mark.parametrize("E,top,groups", [(1, 1, 0), (31, 8, 0), (33, 3, 0), (64, 6, 8), (65, 3, 0), (96, 8, 8), (128, 8, 8), (255, 4, 0),
                                          (256, 32, 16)])
def test_choice_among_few_and_many_experts(E, top, groups):
    """One, two and eight experts per lane: the choice and the weights that float64 gives."""
    z = rnd(37, E, seed=E + 1)
    keep = max(1, groups // 2)
    ids, weights = select(z, top, "all", groups, keep)
    c = z.double()
    if groups:
        best = c.view(37, groups, -1).max(dim=-1).values
        kept = torch.zeros_like(best).scatter_(1, best.topk(keep, dim=1).indices, 1.0).repeat_interleave(E // groups, dim=1)
        c = c.masked_fill(kept == 0, float("-inf"))
    p, want = torch.softmax(z.double(), dim=1), c.topk(top, dim=1).indices
    assert torch.equal(ids.long(), want)
    share = p.gather(1, want)
    share = 1.5 * share / share.sum(dim=1, keepdim=True)
    assert (weights.double() - share).abs().max().item() <= 1e-5

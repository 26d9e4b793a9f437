"""Models whose router leaves out whole groups of experts: their decode steps add up in an order that is kept from one version
of the kernels to the next (``ops.kept_sums``), the other models' need not."""

import threading

import pytest
import torch

import vepevik_configs as V

DEV = "cuda:0"


def ops():
    from mini_infer_b200.csrc import ops as o
    return o


def test_the_scope_is_the_threads_own_and_ends():
    o, seen = ops(), []
    assert not o._sums_kept()
    with o.kept_sums():
        with o.kept_sums():
            pass
        assert o._sums_kept()
        th = threading.Thread(target=lambda: seen.append(o._sums_kept()))
        th.start()
        th.join()
    with pytest.raises(ValueError):
        with o.kept_sums():
            raise ValueError
    assert seen == [False] and not o._sums_kept()


def test_models_with_groups_of_experts_ask_for_it():
    from mini_infer_b200.config import load_config
    from mini_infer_b200.parts.model import DecoderModel

    for which, cfg in V.CONFIGS.items():
        groups = [l["mlp"]["router"].get("groups") for l in cfg["layers"] if l.get("mlp") and l["mlp"]["kind"] == "moe"]
        want = any(g and g["keep"] < g["count"] for g in groups)
        arch, parsed = load_config(cfg)
        assert DecoderModel(arch.assemble(parsed))._keeps_sums == want, which


@pytest.mark.gpu
@pytest.mark.parametrize("which", list(V.CONFIGS))
@pytest.mark.parametrize("graph", [False, True])
def test_decode_steps_take_the_kernels_that_keep_the_order(which, graph, monkeypatch):
    """Single tokens of a model with groups of experts reach neither ``gemm_rows`` nor the tensor-core product of few rows per
    expert nor shorter stretches of keys; those of another model reach ``gemm_rows``."""
    from mini_infer_b200.engine import ModelRunner, StepEntry

    o, cfg = ops(), V.CONFIGS[which]
    state = V.random_state(cfg, seed=3, ranks=V.RANKS[which])
    runner = ModelRunner.from_state_dict(cfg, state, dtype="bfloat16", block_size=V.PAGE_SIZE[which], num_blocks=8,
                                         max_requests=2, cuda_graph=graph)
    calls, kept = [], []
    for name in ("gemm_rows", "gemm_tma"):
        real = getattr(o, name)
        monkeypatch.setattr(o, name, lambda *a, real=real, name=name, **k: (calls.append(name), kept.append(o._sums_kept()), real(*a, **k))[2])
    real_experts = o.moe_experts
    monkeypatch.setattr(o, "moe_experts", lambda *a, **k: (kept.append(o._sums_kept()), real_experts(*a, **k))[1])
    runner.add_request("r")
    runner.step([StepEntry("r", [1, 2, 3], [2])])
    calls.clear(), kept.clear()
    for t in (4, 5):
        runner.step([StepEntry("r", [t], [0])])
    assert len(calls) > 0
    if runner.model._keeps_sums:
        assert "gemm_rows" not in calls and all(kept)
    else:
        assert "gemm_tma" not in calls and not any(kept)


@pytest.mark.gpu
@pytest.mark.parametrize("E,K,H,rows", [(3, 520, 37, 8), (2, 1024, 64, 5), (4, 40, 16, 1), (2, 2048, 24, 3), (1, 264, 1, 2)])
def test_experts_in_the_kept_order_to_the_bit(E, K, H, rows):
    """Lane l of 32 takes k from 8 l, 8 l + 256, ... on, one fused multiply-add after the other, and the lanes' sums are added
    16, 8, 4, 2 and 1 apart: the same steps in the same order on the CPU, the fused multiply-add as a float64 sum of an exact product
    rounded once more (two roundings differ from one only on a tie of 29 zero bits)."""
    a = torch.randn(E * rows, K, generator=torch.Generator().manual_seed(1)).bfloat16()
    w = (torch.randn(E, H, K, generator=torch.Generator().manual_seed(2)) * K ** -0.5).bfloat16()
    plan = torch.tensor([E] + [rows * e for e in range(E + 1)] + [x for e in range(E) for x in (e, rows * e, rows)] + [0] * (3 * E),
                        dtype=torch.int32, device=DEV)
    y = torch.empty(E * rows, H, device=DEV)
    ad, wd = a.to(DEV), w.to(DEV)
    assert ops()._lib("moe").mi_moe_down(ad.data_ptr(), wd.data_ptr(), H * K, plan.data_ptr(), E, y.data_ptr(), E * rows, H, K, 8, 1,
                                         1, torch.cuda.current_stream().cuda_stream) == 0
    prod = (a.double().reshape(E, rows, 1, K) * w.double().reshape(E, 1, H, K)).reshape(E * rows, H, K)
    lanes = torch.nn.functional.pad(prod, (0, -K % 256)).reshape(E * rows, H, -1, 32, 8).permute(0, 1, 3, 2, 4).flatten(3)
    acc = torch.zeros(E * rows, H, 32)
    for i in range(lanes.shape[-1]):
        acc = (acc.double() + lanes[..., i]).float()
    while acc.shape[-1] > 1:
        half = acc.shape[-1] // 2
        acc = acc[..., :half] + acc[..., half:]
    assert torch.equal(y.cpu(), acc[..., 0])


@pytest.mark.gpu
def test_products_inside_the_scope_are_those_of_gemm_tma():
    o = ops()
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(8, 4096, generator=g).bfloat16().to(DEV), (torch.randn(514, 4096, generator=g) / 64).bfloat16().to(DEV)
    with o.kept_sums():
        inside, pairs = o.linear(x, w, torch.float32), o.linear_swiglu(x, w)
    assert torch.equal(inside, o.gemm_tma(x, w, torch.float32)) and torch.equal(pairs, o.gemm_tma(x, w, swiglu=1))
    assert torch.equal(o.linear(x, w, torch.float32), o.gemm_rows(x, w, torch.float32))

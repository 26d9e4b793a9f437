"""Captured steps whose layers have two branches (``parts/streams.py``): the same bits as the steps launched kernel by
kernel, which are one chain, over many replays back to back."""

import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("model,which", [("ruvurax", "P"), ("ruvurax", "M"), ("lilulix", "A")])
def test_two_branches_give_the_bits_of_one_chain(model, which, dtype):
    from mini_infer_b200.engine import StepEntry
    from mini_infer_b200.parts import streams

    module = importlib.import_module(f"test_{model}_gpu")
    cfg, n_new = module.CONFIGS[which], 40
    tokens = [module.prompt(cfg, n + n_new, salt=30 + n) for n in (3, 11, 7)]
    rows, used = {}, []
    real = streams.beside.run

    def run(self, f):
        used.append(self.on)
        return real(self, f)

    streams.beside.run = run
    try:
        for graph in (False, True):
            runner = module.make_runner(which, dtype, num_blocks=64, cuda_graph=graph)
            for i in range(3):
                runner.add_request(i)
            runner.step([StepEntry(i, t[:len(t) - n_new]) for i, t in enumerate(tokens)])
            got = []
            for j in range(n_new):
                step = runner.step([StepEntry(i, [t[len(t) - n_new + j]], [0]) for i, t in enumerate(tokens)])
                got.append(step.logits.clone())
            rows[graph] = torch.stack(got)
            if graph:
                assert any(used), "no branch was recorded"
                assert all(s.replays == n_new - 1 for s in runner.stepper._graphs.values())
            else:
                assert used and not any(used)
    finally:
        streams.beside.run = real
    assert torch.isfinite(rows[True]).all()
    assert torch.equal(rows[True], rows[False])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("requests", [5, 19])
def test_two_branches_of_wider_layers(requests, dtype):
    """Heads of 64 and 128, whose norms and gates run in lanes, and with 19 requests the library's products on both streams: the
    bits of one chain."""
    from mini_infer_b200.engine import ModelRunner, StepEntry

    import ruvurax_configs as C

    both = C.parallel(heads=4, kv_heads=2, dim=64, vdim=64, window=33, rot_dims=64, rot_base=1000.0, scale=0.125, r_heads=2,
                      r_dim=64, r_vdim=128, tau=8.0, left_scale=0.7, right_scale=1.2,
                      mlp=C.experts(8, 2, 64, 0.7, {"ff": 96, "limit": 1.3}))
    cfg = C.config([both, C.rglru(128, 2, 4, C.experts(8, 2, 64, 1.0, {"ff": 64, "limit": 0.5})), both],
                   vocab=101, width=128, scale=0.5, eps=1e-6)
    state, n_new = C.random_state(cfg, seed=5), 12
    lens = [1 + (7 * i) % 23 for i in range(requests)]
    tokens = [[(13 * i + 5 * j + i * j) % 101 for j in range(n + n_new)] for i, n in enumerate(lens)]
    rows = {}
    for graph in (False, True):
        runner = ModelRunner.from_state_dict(cfg, state, dtype=dtype, block_size=16, num_blocks=4 * requests, max_requests=requests,
                                             cuda_graph=graph)
        for i in range(requests):
            runner.add_request(i)
        runner.step([StepEntry(i, t[:n]) for i, (t, n) in enumerate(zip(tokens, lens))])
        got = [runner.step([StepEntry(i, [t[n + j]], [0]) for i, (t, n) in enumerate(zip(tokens, lens))]).logits.clone()
               for j in range(n_new)]
        rows[graph] = torch.stack(got)
    assert torch.isfinite(rows[True]).all() and torch.equal(rows[True], rows[False])


def test_both_branches_asking_for_one_workspace_is_an_error():
    """Found while the step is recorded: nothing runs."""
    from mini_infer_b200.csrc import ops
    from mini_infer_b200.parts import streams

    x, w = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) for s in ((4, 128), (256, 128)))
    want = ops.gemm_tma(x, w).clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(ops.KernelError, match="both branches"):
        with torch.cuda.graph(graph):
            with streams.beside() as side:
                side.run(lambda: ops.gemm_tma(x, w))
                ops.gemm_tma(x, w)
    assert not ops.open_branches() and torch.equal(ops.gemm_tma(x, w), want)

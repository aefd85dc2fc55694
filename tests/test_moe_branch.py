"""Routed experts with a shared expert inside a branch of the caller's: the list has one side stream, and what was accepted without the expert's own branch still is."""
import pytest
import torch

WIDTH, FF, EXPERTS, SHARED, TOP = 24, 16, 5, 12, 2


def weights(device):
    g = torch.Generator().manual_seed(3)
    rnd = lambda *s: (torch.randn(*s, generator=g) * s[-1] ** -0.5).to(device)  # noqa: E731
    return dict(router=rnd(EXPERTS, WIDTH), up=rnd(EXPERTS, FF, WIDTH), down=rnd(EXPERTS, WIDTH, FF), shared_up=rnd(SHARED, WIDTH), shared_down=rnd(WIDTH, SHARED))


def build(device, M, slot, x, out, other, where):
    """where: the expert layer outside of any branch, on the side stream, beside it, or behind an open side stream at the list's end."""
    from qwen3_tts_cuda_graphs_b200.config import MoEFFConfig
    from qwen3_tts_cuda_graphs_b200.seq_ops import StepBuilder

    b, c, w = StepBuilder(torch.device(device), M, slot, True), MoEFFConfig(EXPERTS, 0, TOP, 1, 1, 1.3, FF, SHARED), weights(device)
    experts = lambda: b.moe_ff(x, x, c, w, out)  # noqa: E731
    double = lambda: b.sum_norm(x[None], 1, torch.full((1,), 2.0, device=device), out=other)  # noqa: E731
    if where == "alone":
        double()
        experts()
    else:
        b.branch(0)
        experts() if where == "side" else double()
        b.branch(1)
        double() if where == "side" else experts()
        if where != "end":
            b.branch(2)
    return b.finish()


@pytest.mark.parametrize("where", ["alone", "side", "beside", "end"])
def test_a_list_opens_one_side_stream_at_a_time(where):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    x = torch.zeros(7, WIDTH)
    plan = build("cpu", 7, None, x, torch.zeros(7, WIDTH), torch.zeros(7, WIDTH), where)
    open_, opened = False, 0
    for o in plan.ops:
        if o.kind == K.K_BRANCH:
            assert not (o.i0 == 0 and open_)
            opened += o.i0 == 0
            open_ = o.i0 == 0 or (o.i0 == 1 and open_)
    assert opened == 1      # the expert's own, or the caller's
    assert sum(o.kind == K.K_GEMM for o in plan.ops) == 3 and sum(o.kind == K.K_MOE_COMBINE for o in plan.ops) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 40])
def test_the_same_values_wherever_it_runs(M):
    from qwen3_tts_cuda_graphs_b200 import codec as K
    from qwen3_tts_cuda_graphs_b200.seq_state import SequenceStateManager

    slot = SequenceStateManager([], 100, torch.device("cuda"), 1).acquire("t")
    x = torch.randn(M, WIDTH, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M))
    got = []
    for where in ("alone", "side", "beside", "end"):
        out, other = torch.zeros(M, WIDTH, device="cuda"), torch.zeros(M, WIDTH, device="cuda")
        K.run_op_plan(K.load_lib(), build("cuda", M, slot, x, out, other, where), False)
        torch.cuda.synchronize()
        got.append((out, other))
    assert got[0][0].abs().sum() > 0
    for out, other in got:
        assert torch.equal(out, got[0][0]) and torch.equal(other, 2 * x)

"""A kernel that is launched while the one before it is still running reads that one's results after its wait, never
before: what the earlier kernel writes is poisoned first, so a number fetched too early shows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("parts_width", [512, 256, 128, 1024])
def test_the_gated_norm_waits_for_the_scan(parts_width):
    """The state-space scan leaves multiprocessors free for the first blocks of the norm behind it.  Same arithmetic on
    the same numbers: equal to the last bit to a norm that is launched long after the scan has ended."""
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.ops import kernels as K
    T, H, P, N, groups = 2048, 64, 64, 128, 8
    gen = torch.Generator(device=DEV).manual_seed(3)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=DEV)

    u, z = normal(T, H * P + 2 * groups * N).bfloat16(), normal(T, H * P).bfloat16()
    dt, head, weight = normal(T, H).bfloat16(), torch.zeros(H, device=DEV), normal(H * P)
    state = torch.zeros(1, H, N, P, device=DEV)
    batch = build_step_batch([StepItem("a", [0] * T, 0)], {}, [0], torch.device(DEV), 2, T)
    busy = torch.randn(8192, 8192, device=DEV).bfloat16()
    for _ in range(4):
        y = torch.full((T, H * P), float("nan"), device=DEV)
        state.zero_()
        for _ in range(3):
            torch.mm(busy, busy)              # the host is ahead: the norm is queued before the scan begins
        K.ssm_scan(u, dt, head, head, head, state, batch, groups, out=y)
        got = K.gated_group_rmsnorm(y, z, weight, H * P // parts_width, 1e-6)
        torch.cuda.synchronize()
        assert torch.isfinite(y).all()
        assert torch.equal(got, K.gated_group_rmsnorm(y, z, weight, H * P // parts_width, 1e-6))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [2048, 2050])
def test_the_norm_of_chosen_rows_waits_for_the_choice(dtype, width):
    """The rows are chosen by the kernel before: that of the largest of 60,000 numbers, on few multiprocessors.  Read too early
    they are what lay there, -1, which gives zeros."""
    from prelude_b200.ops import kernels as K
    n, wide = 8, 60000
    gen = torch.Generator(device=DEV).manual_seed(4)
    res, weight = torch.randn(n, width, generator=gen, device=DEV), torch.rand(width, generator=gen, device=DEV) + 0.5
    scores = torch.zeros(n, wide, device=DEV)
    picks = torch.randperm(n, generator=gen, device=DEV)
    scores[torch.arange(n, device=DEV), picks] = 1.0
    zero, counts = torch.zeros(n, device=DEV), torch.zeros(n, dtype=torch.int64, device=DEV)
    want = K.gather_add_rmsnorm(None, res, picks.int(), weight, 1e-6, dtype)
    busy = torch.randn(8192, 8192, device=DEV).bfloat16()
    for _ in range(4):
        rows = torch.full((n,), -1, dtype=torch.int32, device=DEV)
        for _ in range(3):
            torch.mm(busy, busy)              # the host is ahead: the norm is queued before the choice begins
        K.sample(scores, zero, counts, counts, out=rows)
        got = K.gather_add_rmsnorm(None, res, rows, weight, 1e-6, dtype)
        torch.cuda.synchronize()
        assert rows.tolist() == picks.tolist() and torch.equal(got, want)

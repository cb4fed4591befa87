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


@pytest.mark.parametrize("rows", [8, 64])                         # the routers of decode and of prompt steps
@pytest.mark.parametrize("captured", [False, True])
def test_the_experts_second_product_waits_for_the_choices(rows, captured):
    """It reads the choices ahead of its own wait.  They come from a router that lets the next kernel begin at once and has
    8,192-wide rows to go through; until it is done, the choices of the call before, which name experts too, lie there."""
    from prelude_b200.ops import kernels as K
    lib, top, E, N, width, wide = K._l.library(), 4, 64, 1024, 768, 8192
    gen = torch.Generator(device=DEV).manual_seed(6)

    def normal(*shape, scale=1.0):
        return (torch.randn(shape, generator=gen, device=DEV) * scale).bfloat16()

    x, up, down = normal(rows, width), normal(E, N, width, scale=width ** -0.5), normal(E, width, N, scale=N ** -0.5)
    routers = [(normal(rows, wide), normal(E, wide, scale=wide ** -0.5)) for _ in range(2)]
    ids, weights = torch.zeros(rows, top, dtype=torch.int32, device=DEV), torch.zeros(rows, top, device=DEV)
    assert K.moe_streams(up, rows * top) and K.moe_streams(down, rows * top)

    def route(n):
        z, w = routers[n % 2]
        rest = (None, None, rows, E, top, 1, 1, 1, 0, 0, 0.0, 1.0, ids.data_ptr(), weights.data_ptr())
        if rows < 64:
            assert lib.pb_moe_route_few(z.data_ptr(), wide, w.data_ptr(), K.dtype_code(z.dtype), wide, *rest, K._stream()) == 0
        else:
            assert lib.pb_moe_route_tokens(z.data_ptr(), wide, w.data_ptr(), wide, *rest, None, K._stream()) == 0

    def products(settled):
        h = K.moe_gemv(x, up, ids, False, torch.bfloat16, act=K.ACT_RELU2)
        return K.moe_gemv(h, down, ids, True, torch.float32, settled=settled)

    want, choices = [], []
    for n in range(2):
        route(n)
        torch.cuda.synchronize()
        choices.append(ids.clone())
        want.append(products(False))
    assert not torch.equal(*choices)

    def steps():
        out = []
        for n in range(8):
            route(n)
            out.append(products(True))
        return out

    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = steps()
    busy = torch.randn(8192, 8192, device=DEV).bfloat16()
    for _ in range(4):
        for _ in range(3):
            torch.mm(busy, busy)              # the host is ahead: all are queued before the first router begins
        if captured:
            graph.replay()
        else:
            got = steps()
        torch.cuda.synchronize()
        for n, y in enumerate(got):
            assert torch.equal(y, want[n % 2])

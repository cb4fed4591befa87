"""The products that stream their weights, where their plan changes: chunks of K, stages, few rows of K, experts with more rows than fit at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=1, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * scale).bfloat16()


# rows x K: one chunk with many stages, four; two chunks; 1,024-element chunks beside 16 rows; 640; three stages; two; one set of sums; three stages of
# parts, short pieces of parts; N: all of a block's rows in the ring at once, and not
@pytest.mark.parametrize("M,K_", [(1, 48), (8, 1024), (8, 2560), (16, 2560), (2, 4096), (8, 4096), (16, 4096), (12, 5120), (16, 5120), (8, 8192), (2, 12288), (16, 6160),
                                  (16, 6144), (1, 20000), (2, 49600), (11, 8192), (8, 9728), (14, 6912)])
@pytest.mark.parametrize("N", [9, 700, 3000])
def test_stream_plans(M, K_, N):
    from prelude_b200.ops.linear import gemm_stream, stream_takes, tc_status
    x, w = rnd(M, K_), rnd(N, K_, seed=2, scale=K_ ** -0.5)
    assert stream_takes(x, w)
    want = x.double() @ w.double().T
    got = gemm_stream(x, w, out_dtype=torch.float32)
    # products exact in float32; a chain adds K / 512 steps of 16, each cut to 2^-23 of the sum so far, then 4 chains and 8 warps are added
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -23 * (K_ / 512 + 16)
    assert torch.equal(gemm_stream(x, w, out_dtype=torch.float32), got) and int(tc_status(x.device)) == 0


# steps whose rows are fetched whole beside few rows of x, and in pieces beside many; pieces in whole turns over the chains and not
@pytest.mark.parametrize("few,many,K_", [(2, 12, 2432), (2, 16, 2432), (8, 12, 2560), (1, 16, 2560), (2, 8, 3072), (1, 14, 3072), (2, 11, 4096), (8, 14, 4096), (1, 9, 5120),
                                         (2, 14, 6144), (1, 6, 8192), (1, 2, 12288)])
def test_sums_do_not_depend_on_how_k_is_fetched(few, many, K_):
    from prelude_b200.ops.linear import gemm_stream
    x, w = rnd(many, K_), rnd(3000, K_, seed=2, scale=K_ ** -0.5)
    got = gemm_stream(x, w, out_dtype=torch.float32)
    assert torch.equal(gemm_stream(x[:few], w, out_dtype=torch.float32), got[:few])
    assert torch.equal(gemm_stream(x, w[:9], out_dtype=torch.float32), got[:, :9])


@pytest.mark.parametrize("gated,act", [(False, "NONE"), (False, "RELU2"), (True, "NONE"), (True, "CLAMPED")])
@pytest.mark.parametrize("slots", [False, True])
@pytest.mark.parametrize("T,top,E,N,K_", [(1, 1, 1, 8, 768), (1, 4, 32, 100, 1040), (2, 2, 4, 136, 2048), (8, 4, 32, 2048, 2048), (9, 2, 3, 24, 4096), (17, 1, 2, 40, 2416),
                                          (16, 6, 64, 512, 4096), (40, 8, 256, 64, 768), (24, 2, 2, 300, 7168), (3, 8, 1024, 16, 784)])
def test_experts_streamed(T, top, E, N, K_, gated, act, slots):
    from prelude_b200.ops import kernels as K
    from prelude_b200.ops import library
    assert library.library().pb_moe_stream_supported(K_, T * top, E)
    w = rnd(E, N * (2 if gated else 1), K_, scale=K_ ** -0.5)
    a = rnd(T * top if slots else T, K_, seed=3)
    g = torch.Generator(device=DEV).manual_seed(5)
    ids = torch.stack([torch.randperm(E, generator=g, device=DEV)[:top] for _ in range(T)]).int()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kw = dict(gated=gated, act=getattr(K, "ACT_" + act), limit=2.0, alpha=1.7, status=status)
    got = K.moe_gemv(a, w, ids, slots, torch.float32, **kw)
    rows, want = (a if slots else a.repeat_interleave(top, 0)).double(), torch.empty(T * top, N, dtype=torch.float64, device=DEV)
    for e in ids.unique().tolist():
        m = (ids.flatten() == e).nonzero().flatten()
        z = rows[m] @ w[e].double().T
        if gated:
            u = z[:, N:]
            z = z[:, :N]
            z = torch.nn.functional.silu(z) * u if act == "NONE" else z.clamp(max=2.0) * torch.sigmoid(1.7 * z.clamp(max=2.0)) * (u.clamp(-2, 2) + 1)
        elif act == "RELU2":
            z = torch.relu(z) ** 2
        want[m] = z
    # Steps of sixteen products cut to 2^-23 of the largest (2^-24 in the root mean square); a chain adds K / 512 of them, four chains meet, the warps'
    # sums are added in 64 bits: that many sums rounded by 2^-25 of themselves, a chain's early ones of less.  Activations: a product of two such sums, or more
    most = 2.0 ** -25 * (4 + (K_ / 512 + 1) / 2 + 3) ** 0.5
    assert float((got.double() - want).norm() / want.norm()) < (most if act == "NONE" and not gated else 4 * most)
    assert int(status) == 0 and torch.equal(K.moe_gemv(a, w, ids, slots, torch.float32, **kw), got)
    # one rounding to bfloat16
    assert torch.equal(K.moe_gemv(a, w, ids, slots, torch.bfloat16, **kw), got.bfloat16())
    if not slots and T > 1:                          # a token's result does not depend on who else chose its experts
        assert torch.equal(K.moe_gemv(a[1:2], w, ids[1:2].contiguous(), False, torch.float32, **kw), got[top:2 * top])


# one expert with many rows beside others with few: its eights are dealt like experts
@pytest.mark.parametrize("T,top,E,N,K_", [(9, 1, 3, 40, 768), (40, 8, 33, 264, 1040), (64, 8, 64, 136, 2048), (128, 4, 1024, 24, 784), (100, 2, 2, 700, 4096)])
def test_experts_with_many_rows(T, top, E, N, K_):
    from prelude_b200.ops import kernels as K
    w, a = rnd(E, N, K_, scale=K_ ** -0.5), rnd(T, K_, seed=3)
    g = torch.Generator(device=DEV).manual_seed(7)
    ids = torch.stack([torch.randperm(E, generator=g, device=DEV)[:top] for _ in range(T)]).int()
    hot = E // 2
    ids[: T - 3, 0] = torch.where((ids[: T - 3] == hot).any(1), ids[: T - 3, 0], hot)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = K.moe_gemv(a, w, ids, False, torch.float32, status=status)
    for t in range(T):                               # each token's result is what it is alone
        assert torch.equal(K.moe_gemv(a[t:t + 1], w, ids[t:t + 1].contiguous(), False, torch.float32), got[t * top:t * top + top])
    want = torch.stack([w[e].double() @ a[i // top].double() for i, e in enumerate(ids.flatten().tolist())])
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -25 * (4 + (K_ / 512 + 1) / 2 + 3) ** 0.5 and int(status) == 0


# a pair, the second of which reads the choices before the first has ended: resident rows, rows that move, blocks without a share
@pytest.mark.parametrize("T,top,E,N,K_", [(1, 1, 2, 768, 784), (8, 4, 32, 2048, 2048), (40, 8, 64, 1024, 768), (3, 8, 1024, 800, 1040)])
def test_second_product_begins_early(T, top, E, N, K_):
    from prelude_b200.ops import kernels as K
    up, down, x = rnd(E, N, K_, scale=K_ ** -0.5), rnd(E, K_, N, seed=2, scale=N ** -0.5), rnd(T, K_, seed=3)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def pair(n, settled):
        ids = (torch.arange(T * top, device=DEV, dtype=torch.int32).view(T, top) * 7 + n) % E     # new choices just ahead
        h = K.moe_gemv(x, up, ids, False, torch.bfloat16, act=K.ACT_RELU2, status=status)
        return K.moe_gemv(h, down, ids, True, torch.float32, status=status, settled=settled)

    want = [pair(n, False) for n in range(8)]
    got = [pair(n, True) for n in range(8)]
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    # ids that name no expert leave every block without a share
    none = torch.full((T, top), -1, dtype=torch.int32, device=DEV)
    h = K.moe_gemv(x, up, none, False, torch.bfloat16, act=K.ACT_RELU2, status=status)
    K.moe_gemv(torch.zeros_like(h), down, none, True, torch.float32, status=status, settled=True)
    assert int(status) == 0

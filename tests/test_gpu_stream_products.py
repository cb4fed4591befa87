"""The products that stream their weights, where their plan changes: chunks of K, stages, few rows of K, experts with more rows than fit at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=1, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * scale).bfloat16()


# rows x K: one chunk with many stages, four; two chunks; 1,024-element chunks beside 16 rows; 640; three stages; two; one set of sums
@pytest.mark.parametrize("M,K_", [(1, 48), (8, 1024), (8, 2560), (16, 2560), (2, 4096), (8, 4096), (16, 4096), (12, 5120), (16, 5120), (8, 8192), (2, 12288), (16, 6400),
                                  (16, 6144), (1, 20000), (2, 49600)])
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

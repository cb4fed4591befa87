"""The causal convolution in runs of tokens: every way a run can meet a sequence's start, its end and the step's end, padding
rows, and the carried inputs, moved on by the same kernel (one token a sequence) or by one of their own."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _plain(x, w, bias, carried, lens):
    """[T, C] in float64, the sum of its terms' magnitudes, and the carried inputs behind the step."""
    out, size, after, at = [], [], [], 0
    for r, n in enumerate(lens):
        rows = torch.cat([carried[r], x[at:at + n]]).double()
        K = w.shape[1]
        acc = sum(rows[j:j + n] * w[:, j].double() for j in range(K))
        size.append(sum((rows[j:j + n] * w[:, j].double()).abs() for j in range(K)) + bias.double().abs())
        acc = acc + bias.double()
        out.append(acc * torch.sigmoid(acc))
        after.append(torch.cat([carried[r], x[at:at + n]])[-(K - 1):])
        at += n
    return torch.cat(out), torch.cat(size), torch.stack(after)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps", [2, 3, 4, 5])
@pytest.mark.parametrize("lens", [[72], [65], [8, 56, 9, 7, 1, 2, 90], [1, 1, 1, 70], [1], [1] * 70, [3, 2, 1]])
@pytest.mark.parametrize("channels", [64, 1000, 12])
def test_convolution_and_carried_inputs(dtype, taps, lens, channels):
    """Every term and sum is rounded to float32 once (6e-8 of the terms' magnitudes, which SiLU's slope of at most 1.1 passes
    on), SiLU adds a few roundings of its own, and the result is rounded to its type (bfloat16 has eight bits: 2^-8 of the value)."""
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.ops import kernels as K
    gen = torch.Generator(device=DEV).manual_seed(11)
    T, R = sum(lens), len(lens)
    x = torch.randn(T, channels + 16, generator=gen, device=DEV).to(dtype)[:, :channels]
    w, bias = torch.randn(channels, taps, generator=gen, device=DEV), torch.randn(channels, generator=gen, device=DEV)
    carried = torch.randn(R, taps - 1, channels, generator=gen, device=DEV).to(dtype)
    want, size, after = _plain(x, w, bias, carried, lens)
    batch = build_step_batch([StepItem(i, [0] * n, 5 * i) for i, n in enumerate(lens)], {}, list(range(R))[::-1], torch.device(DEV), 2, 1 << 20)
    held = carried.flip(0).contiguous()                    # request i lies in slot R - 1 - i
    got = K.causal_conv_silu(x, w, bias, held, batch, advance=batch.decode_only)
    if not batch.decode_only:
        K.conv_state_update(x, held, batch)
    bound = 1.1 * (taps + 1) * 6e-8 * size + (4 * 6e-8 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)) * want.abs() + 1e-12
    assert bool(((got.double() - want).abs() <= bound).all())
    assert torch.equal(held.flip(0), after)

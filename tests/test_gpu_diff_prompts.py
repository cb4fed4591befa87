"""Differential attention of prompt portions on the tcgen05 kernel: portions that end inside a block, a tile and a page, contexts before them,
windows, single tokens beside them, every page size and group it takes, values of 64 and 128, rests of pages that hold NaN; against float64."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def case(shape, H, G, vdim, page, window, gated=True, seed=0):
    from prelude_b200.cache.manager import CacheManager
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.ops import kernels as K
    from prelude_b200.parts.registry import KvPagesNeed
    dev, dim = torch.device(DEV), 64
    g = torch.Generator(device=DEV).manual_seed(seed)
    cache = CacheManager([KvPagesNeed(2 * G, dim, None, v_heads=G, v_head_dim=vdim)], page, sum(-(-(a + b) // page) for a, b in shape) + 3, len(shape), dev, torch.bfloat16)
    mine = cache.layer_cache(0)
    mine.k_pages.fill_(float("nan"))
    mine.v_pages.fill_(float("nan"))
    for r, (have, new) in enumerate(shape):
        cache.add_request(r)
        cache.grow(r, have + new)
    slots = [cache.slot_of(r) for r in range(len(shape))]
    keys, values = [], []
    for r, (have, new) in enumerate(shape):
        n = have + new
        keys.append(torch.randn(n, G * 2 * dim, generator=g, device=DEV).bfloat16())
        values.append(torch.randn(n, G * vdim, generator=g, device=DEV).bfloat16())
        b = build_step_batch([StepItem(r, [0] * n, 0)], cache.block_tables([r]), [slots[r]], dev, 2, 1 << 20)
        K.kv_write_pages(keys[r], values[r], mine.k_pages, mine.v_pages, b.positions, b.table_row_of_token, b.block_tables[0], b.status)
    batch = build_step_batch([StepItem(r, [0] * new, have) for r, (have, new) in enumerate(shape)], cache.block_tables(list(range(len(shape)))), slots, dev, 2, 1 << 20)
    T = batch.n_tokens
    proj = torch.randn(T, H * 2 * dim + H * vdim + 8, generator=g, device=DEV).bfloat16()
    q, gate = proj[:, :H * 2 * dim], proj[:, H * 2 * dim + 8:] if gated else None
    spec = SimpleNamespace(num_heads=H, num_kv_heads=G, head_dim=dim, value_dim=vdim, softmax_scale=dim ** -0.5, lambda_init=0.5, norm_eps=1e-6,
                           query_temperature=SimpleNamespace(coef=0.2, every=32), window=window)
    return q, gate, keys, values, batch, mine, spec, cache


def plain(q, gate, keys, values, shape, spec, lam):
    H, G, d, e = spec.num_heads, spec.num_kv_heads, spec.head_dim, spec.value_dim
    out, at = [], 0
    for (have, new), k, v in zip(shape, keys, values):
        n = have + new
        i, j = torch.arange(have, n, device=DEV).view(-1, 1), torch.arange(n, device=DEV).view(1, -1)
        hidden = (j > i) | ((i - j >= spec.window) if spec.window else (j > i))
        tau = (1 + 0.2 * torch.log(((i + 1) // 32 + 1).double())).view(1, new, 1)
        qq = q[at:at + new].double().reshape(new, H, 2, d)
        kk, vv = k.double().view(n, G, 2, d).repeat_interleave(H // G, 1), v.double().view(n, G, e).repeat_interleave(H // G, 1)
        maps = [torch.einsum("hij,jhe->ihe", torch.softmax((torch.einsum("ihd,jhd->hij", qq[:, :, c], kk[:, :, c]) * d ** -0.5 * tau).masked_fill(hidden, -1e300), -1), vv)
                for c in (0, 1)]
        o = maps[0] - lam * maps[1]
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * 0.5
        if gate is not None:
            o = o * torch.sigmoid(gate[at:at + new].double().reshape(new, H, e))
        out.append(o)
        at += new
    return torch.cat(out)


@pytest.mark.parametrize("shape", [[(0, 1)], [(0, 129)], [(127, 2), (128, 1)], [(0, 700)], [(300, 65), (5, 1), (0, 31), (600, 200)]])
@pytest.mark.parametrize("H,G,vdim,page", [(16, 4, 128, 16), (8, 8, 64, 8), (16, 1, 128, 32), (4, 2, 128, 128), (2, 1, 64, 256), (8, 1, 128, 64)])
@pytest.mark.parametrize("window", [None, 100])
def test_against_float64(shape, H, G, vdim, page, window):
    from prelude_b200.ops import diff_attention as D
    q, gate, keys, values, batch, mine, spec, _ = case(shape, H, G, vdim, page, window, seed=H + vdim)
    assert D._l.library().pb_diff_attention_tcgen05_supported(H, G, 64, vdim, page, q.stride(0), q.data_ptr(), gate.stride(0), gate.data_ptr())
    batch.decode_only = False                    # single tokens too: as they lie beside a portion
    for ga in (gate, None):
        got = D.diff_attention(q, ga, mine.k_pages, mine.v_pages, batch, 0, spec, 0.3)
        want = plain(q, ga, keys, values, shape, spec, 0.3)
        # the rounding of the result, 2^-9 at most and 1.7e-3 in the 2-norm; scores, weights (16 bits in two parts) and sums add 1e-4
        assert float((got.double() - want).norm() / want.norm()) < 2.2e-3
        assert torch.equal(D.diff_attention(q, ga, mine.k_pages, mine.v_pages, batch, 0, spec, 0.3), got)
    assert int(batch.status) == 0


def test_maxima_that_grow_and_fall():
    # scores that rise and fall by far more than the kernel lets a maximum grow before it rescales
    from prelude_b200.ops import diff_attention as D
    shape = [(0, 900)]
    q, gate, keys, values, batch, mine, spec, cache = case(shape, 4, 2, 128, 16, None, seed=3)
    from prelude_b200.ops import kernels as K
    q[:, ::64] = 4.0
    ramp = torch.arange(900, device=DEV).float() / 50
    keys[0][:, 0], keys[0][:, 64] = ramp.bfloat16(), (-ramp).bfloat16()
    keys[0][:, 128], keys[0][:, 192] = torch.sin(ramp * 3).bfloat16() * 16, ramp.bfloat16() * 2
    K.kv_write_pages(keys[0], values[0], mine.k_pages, mine.v_pages, batch.positions, batch.table_row_of_token, batch.block_tables[0], batch.status)
    got = D.diff_attention(q, gate, mine.k_pages, mine.v_pages, batch, 0, spec, 0.3)
    want = plain(q, gate, keys, values, shape, spec, 0.3)
    assert float((got.double() - want).norm() / want.norm()) < 2.2e-3


def test_calls_that_keep_the_other_kernel():
    from prelude_b200.ops import diff_attention as D
    takes = D._l.library().pb_diff_attention_tcgen05_supported
    assert takes(16, 4, 64, 128, 16, 4096, 1 << 20, 4096, 1 << 20) and takes(16, 4, 64, 128, 16, 4096, 1 << 20, 0, None)
    for bad in ((6, 2, 64, 128, 16, 4096, 1 << 20, 0, None), (32, 1, 64, 128, 16, 4096, 1 << 20, 0, None), (16, 4, 128, 128, 16, 4096, 1 << 20, 0, None),
                (16, 4, 64, 96, 16, 4096, 1 << 20, 0, None), (16, 4, 64, 128, 12, 4096, 1 << 20, 0, None), (16, 4, 64, 128, 48, 4096, 1 << 20, 0, None),
                (16, 4, 64, 128, 16, 4100, 1 << 20, 0, None), (16, 4, 64, 128, 16, 4096, (1 << 20) + 8, 0, None), (16, 4, 64, 128, 16, 4096, 1 << 20, 4100, 1 << 20)):
        assert not takes(*bad)


@pytest.mark.parametrize("scale,offset", [(-0.125, 0), (0.0, 0), (0.125, 4), (-0.125, 2)])
def test_scales_and_results_that_keep_the_other_kernel(monkeypatch, scale, offset):
    # a scale that is not positive, a result that is not 16-byte aligned: taken before there was a tcgen05 kernel, and still
    from prelude_b200.ops import diff_attention as D
    shape = [(40, 100), (0, 20)]
    q, gate, keys, values, batch, mine, spec, _ = case(shape, 4, 2, 128, 16, None, seed=7)
    spec.softmax_scale = scale
    room = torch.zeros(q.shape[0] * 4 * 128 + offset, dtype=torch.bfloat16, device=DEV)
    out = room[offset:].view(q.shape[0], 4, 128)
    got = D.diff_attention(q, gate, mine.k_pages, mine.v_pages, batch, 0, spec, 0.3, out)
    monkeypatch.setattr(D, "KERNEL", "mma")
    assert got.data_ptr() == out.data_ptr() and torch.equal(got, D.diff_attention(q, gate, mine.k_pages, mine.v_pages, batch, 0, spec, 0.3))
    want = plain(q * (scale / 0.125), gate, keys, values, shape, spec, 0.3)         # (exact: -1, 0 or 1, and 64 ** -0.5 is 0.125)
    # weights rounded to bfloat16 once, 2^-9 each, and the difference of two maps is smaller than either: four times the rounding of the result
    assert float((got.double() - want).norm() / want.norm()) < 4 * 2.2e-3
    assert int(batch.status) == 0

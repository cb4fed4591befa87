"""The tcgen05 prompt attention where the four warps of a row tile have unequal work in many key tiles running: scores beyond half the cap, and
maxima that grow by more than 2^8 from tile to tile, in the 32 rows of one warp alone; over pages and over dense rows, with and without a
window; against float64, and twenty times the same."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
SHAPE = [(2048, 512), (0, 700), (1100, 131)]             # (tokens before the portion, its tokens)


def operands(H, G, kd, vd, slow, seed, slow_head=0):
    """Queries whose rows of one warp are slow: 32 tokens out of 128 (a block has 256 / (H / G) tokens of a head) of one head."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    ks = [torch.randn(a + b, G, kd, generator=g, device=DEV) for a, b in SHAPE]
    vs = [torch.randn(a + b, G, vd, generator=g, device=DEV).bfloat16() for a, b in SHAPE]
    q = torch.randn(sum(b for _, b in SHAPE), H, kd, generator=g, device=DEV)
    scale, at = kd ** -0.5, 0
    for (_, new), k in zip(SHAPE, ks):
        mine = (torch.arange(new, device=DEV) // 32 % 4 == 1).nonzero()[:, 0] + at
        if slow == "cap":
            if at == 0:
                q *= 0.3                             # (scores of a deviation of 0.3: half of the cap, 2, is out of reach)
            q[mine, slow_head] *= 5.0
        else:
            # along one direction the keys climb for eight tiles of 64 and are level for eight, over and over: a step of 2^10 a tile in the
            # slow rows, nothing in the others
            q[..., 0] = 0.0
            q[mine, slow_head, 0] = 8.0 / scale
            k[..., 0] = (torch.arange(k.shape[0], device=DEV) % 1024).clamp(max=512).unsqueeze(1) / 64.0 * 10.0 * math.log(2.0) / 8.0
        at += new
    return q.bfloat16(), [k.bfloat16() for k in ks], vs, scale


def plain(q, ks, vs, scale, window, cap, sink, gate):
    out, big, at = [], [], 0
    H = q.shape[1]
    for (have, new), k, v in zip(SHAPE, ks, vs):
        n, rep = have + new, H // k.shape[1]
        s = torch.einsum("ihd,jhd->hij", q[at:at + new].double(), k.double().repeat_interleave(rep, 1)) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        i, j = torch.arange(have, n, device=DEV).view(-1, 1), torch.arange(n, device=DEV).view(1, -1)
        s = s.masked_fill((j > i) | ((i - j >= window) if window else (j > i)), float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink.double().view(H, 1, 1).expand(H, new, 1)], -1)
        w = torch.softmax(s, -1)[..., :n]
        vv = v.double().repeat_interleave(rep, 1)
        f = 1.0 if gate is None else torch.sigmoid(gate[at:at + new].double()).unsqueeze(-1)
        out.append(torch.einsum("hij,jhe->ihe", w, vv) * f)
        big.append(torch.einsum("hij,jhe->ihe", w, vv.abs()) * f)
        at += new
    return torch.cat(out), torch.cat(big)


def agrees(got, want, big):
    # weights and results rounded to bfloat16 once each, 2^-9 of the sums of absolute values and of the result; float32 scores of up to 110 and the
    # capped scores' polynomial (5e-6 of up to 12) move a weight by less than 1e-4
    return bool(((got.double() - want).abs() <= 2.0 ** -8 * (big + want.abs()) + 1e-4 * big + 1e-6).all())


def paged(G, page, kd, vd, ks, vs, permuted):
    from prelude_b200.cache.manager import CacheManager
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.ops import kernels as K
    from prelude_b200.parts.registry import KvPagesNeed
    dev = torch.device(DEV)
    cache = CacheManager([KvPagesNeed(G, kd, None, v_heads=G, v_head_dim=vd)], page, sum(-(-(a + b) // page) for a, b in SHAPE) + 3, len(SHAPE), dev, torch.bfloat16)
    lc = cache.layer_cache(0)
    lc.k_pages.fill_(float("nan"))
    lc.v_pages.fill_(float("nan"))
    for r, (have, new) in enumerate(SHAPE):
        cache.add_request(r)
        cache.grow(r, have + new)
    slots = [cache.slot_of(r) for r in range(len(SHAPE))]
    for r, (k, v) in enumerate(zip(ks, vs)):
        n = k.shape[0]
        b = build_step_batch([StepItem(r, [0] * n, 0)], cache.block_tables([r]), [slots[r]], dev, 2, 1 << 20)
        if permuted:
            K.kv_write_pages(k.reshape(n, -1), v.reshape(n, -1), lc.k_pages, lc.v_pages, b.positions, b.table_row_of_token, b.block_tables[0], b.status)
        else:
            j = torch.arange(n, device=DEV)
            ids = b.block_tables[0][0].long()[j // page]
            lc.k_pages[ids, :, j % page] = k
            lc.v_pages[ids, :, j % page] = v
    batch = build_step_batch([StepItem(r, [0] * new, have) for r, (have, new) in enumerate(SHAPE)], cache.block_tables(list(range(len(SHAPE)))), slots, dev, 2, 1 << 20)
    return batch, lc, cache


def check(call, batch, want, big):
    first = call().clone()
    assert int(batch.status.item()) == 0
    assert agrees(first, want, big), float((first.double() - want).abs().max())
    for _ in range(20):
        assert torch.equal(call(), first)
    assert int(batch.status.item()) == 0


@pytest.mark.parametrize("H,G,page", [(2, 2, 16), (4, 2, 64), (16, 2, 16)])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window", [None, 700])
def test_growing_maxima_in_one_warp_over_permuted_pages(monkeypatch, H, G, page, dim, window):
    from prelude_b200.ops import attention
    monkeypatch.setattr(attention, "PREFILL_KERNEL", "tc")
    q, ks, vs, scale = operands(H, G, dim, dim, "growing", H + dim, H - 1)
    batch, lc, _cache = paged(G, page, dim, dim, ks, vs, True)
    want, big = plain(q, ks, vs, scale, window, None, None, None)
    check(lambda: attention.paged_attention(q, lc.k_pages, lc.v_pages, batch, 0, scale, window), batch, want, big)


@pytest.mark.parametrize("slow", ["cap", "growing"])
@pytest.mark.parametrize("H,G,page", [(2, 2, 16), (4, 2, 64), (16, 2, 16)])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window", [None, 700])
def test_one_slow_warp_over_pages_with_cap_sink_and_gate(slow, H, G, page, dim, window):
    from prelude_b200.ops import paged_general as PG
    q, ks, vs, scale = operands(H, G, dim, dim, slow, 3 * H + dim)
    batch, lc, _cache = paged(G, page, dim, dim, ks, vs, False)
    cap = 4.0 if slow == "cap" else None
    sink = torch.linspace(-1.0, 2.0, H, device=DEV)
    gate = torch.randn(q.shape[0], H + 3, generator=torch.Generator(device=DEV).manual_seed(9), device=DEV).bfloat16()[:, :H]
    want, big = plain(q, ks, vs, scale, window, cap, sink, gate)
    check(lambda: PG.attention_general(q, lc.k_pages, lc.v_pages, dim, batch, 0, scale, window, sink, softcap=cap, gate=gate), batch, want, big)


@pytest.mark.parametrize("kd,vd", [(64, 64), (128, 128), (192, 128)])
@pytest.mark.parametrize("window", [None, 700])
def test_growing_maxima_in_one_warp_over_dense_rows(kd, vd, window):
    from prelude_b200.ops import paged_general as PG
    H = 2
    q, ks, vs, scale = operands(H, H, kd, vd, "growing", kd, 1)
    batch, _lc, _cache = paged(H, 16, 64, 64, [k[..., :64] for k in ks], [v[..., :64] for v in vs], False)
    plan = PG.rows_plan(batch, window)
    kv = torch.zeros(plan.n_blocks * PG.ROW_BLOCK, H, kd + vd, dtype=torch.bfloat16, device=DEV)
    for b, (r, p0) in enumerate(zip(plan.block_seq.tolist(), plan.block_pos0.tolist())):
        n = min(PG.ROW_BLOCK, ks[r].shape[0] - p0)
        kv[b * PG.ROW_BLOCK:b * PG.ROW_BLOCK + n] = torch.cat([ks[r][p0:p0 + n], vs[r][p0:p0 + n]], -1)
    want, big = plain(q, ks, vs, scale, window, None, None, None)
    out = torch.zeros(q.shape[0], H, vd, dtype=torch.bfloat16, device=DEV)
    check(lambda: PG.attention_rows(q, kv.view(kv.shape[0], -1), vd, batch, plan, scale, None, None, out), batch, want, big)

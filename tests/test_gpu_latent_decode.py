"""Single tokens over a latent that is key and value at once, on the tcgen05 kernel: contexts that end inside a tile and a page, windows that
begin inside one, every number of parts, pages that are not there, what another request left in a page's rest, sinks and gates, padding
rows; against float64."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def make(contexts, H, kd, vd, page, G=1, seed=0, padding=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    per = max(-(-c // page) for c in contexts)
    num_pages = sum(-(-c // page) for c in contexts) + 2
    pages = torch.randn(num_pages, G, page, kd, generator=g, device=DEV).bfloat16()
    order = torch.randperm(num_pages, generator=torch.Generator().manual_seed(seed)).tolist()
    table = torch.full((len(contexts), per), -1, dtype=torch.int32)
    at = 0
    for r, c in enumerate(contexts):
        for b in range(-(-c // page)):
            table[r, b] = order[at]
            at += 1
        if c % page:                             # the rest of the last page: a NaN of somebody else's
            pages[table[r, c // page], :, c % page:] = float("nan")
    T = len(contexts) + padding
    q = torch.randn(T, H, kd, generator=g, device=DEV).bfloat16()
    positions = torch.tensor([c - 1 for c in contexts] + [0] * padding, dtype=torch.int32, device=DEV)
    rows = torch.tensor(list(range(len(contexts))) + [-1] * padding, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(decode_only=True, block_tables={0: table.to(DEV)}, positions=positions, table_row_of_token=rows, max_kv_len=max(contexts),
                            status=torch.zeros(1, dtype=torch.int32, device=DEV), extras={}, n_tokens=T)
    return q, pages, batch


def plain(q, pages, batch, vd, scale, window, sink, gate):
    page, G = pages.shape[2], pages.shape[1]
    T, H, _ = q.shape
    out = torch.zeros(T, H, vd, dtype=torch.float64, device=DEV)
    big = torch.zeros(T, H, 1, dtype=torch.float64, device=DEV)
    for t in range(T):
        r = int(batch.table_row_of_token[t])
        if r < 0:
            continue
        pos = int(batch.positions[t])
        lo = max(0, pos - window + 1) if window else 0
        j = torch.arange(lo, pos + 1, device=DEV)
        ids = batch.block_tables[0][r][j // page].long()
        j, ids = j[ids >= 0], ids[ids >= 0]
        for g in range(G):
            k = pages[ids, g, j % page].double()
            hs = slice(g * H // G, (g + 1) * H // G)
            s = q[t, hs].double() @ k.T * scale
            if sink is not None:
                s = torch.cat([s, sink[hs].double().unsqueeze(1)], 1)
            w = torch.softmax(s, -1)[:, :k.shape[0]]
            out[t, hs] = w @ k[:, :vd]
            big[t, hs] = (w @ k[:, :vd].abs()).amax(-1, keepdim=True)
    if gate is not None:
        out, big = out * torch.sigmoid(gate.double()).unsqueeze(-1), big * torch.sigmoid(gate.double()).unsqueeze(-1)
    return out, big


# the result rounded to bfloat16 (2^-9 of it), weights too on the general kernel (2^-9 of sums of size `big`), scores of size ~6 from float32
# sums of 576 products (1e-5)
def agrees(got, want, big):
    return bool(((got.double() - want).abs() <= 2.0 ** -8 * (big + want.abs()) + 1e-4).all())


@pytest.mark.parametrize("contexts", [[1], [63, 64, 65], [3000, 17, 128, 1000, 2], [700] * 20, [129] * 150])
@pytest.mark.parametrize("H,kd,vd,page,G", [(32, 576, 512, 16, 1), (16, 576, 512, 16, 1), (4, 192, 128, 8, 1), (40, 320, 256, 32, 1), (24, 256, 128, 64, 2)])
@pytest.mark.parametrize("window", [0, 100])
def test_against_float64(contexts, H, kd, vd, page, G, window):
    from prelude_b200.ops import paged_general as PG
    q, pages, batch = make(contexts, H, kd, vd, page, G, seed=len(contexts) + H, padding=2)
    scale = 2.0 * kd ** -0.5
    gen = torch.Generator(device=DEV).manual_seed(3)
    sink = torch.randn(H, generator=gen, device=DEV)
    gate = torch.randn(q.shape[0], H + 8, generator=gen, device=DEV).bfloat16()[:, :H]
    assert PG.latent_takes(q, pages, None, vd, batch, 0, None, None)
    for sk, ga in ((None, None), (sink, gate)):
        want, big = plain(q, pages, batch, vd, scale, window, sk, ga)
        for parts in (0, 1, 2, 3, 8):
            out = torch.full((q.shape[0], H, vd), 7.0, dtype=torch.bfloat16, device=DEV)
            PG.attention_latent(q, pages, vd, batch, 0, scale, window, sk, ga, out, parts)
            n = len(contexts)
            assert agrees(out[:n], want[:n], big[:n]), (parts, float((out[:n].double() - want[:n]).abs().max()))
            assert bool((out[n:] == 7).all())                     # padding rows are left alone
    assert int(batch.status) == 0


def test_scores_that_grow_and_fall():
    # maxima that grow by much more than the kernel's threshold tile after tile, that fall, and rows whose first tiles weigh nothing
    from prelude_b200.ops import paged_general as PG
    H, kd, vd = 32, 576, 512
    q, pages, batch = make([1000, 1000, 1000], H, kd, vd, 16, seed=5)
    table = batch.block_tables[0]
    q[:, :, 0] = 1.0
    for r, slope in enumerate((0.2, -0.2, 1.0)):
        for j in range(1000):
            pages[table[r, j // 16], 0, j % 16, 0] = slope * j if r < 2 else (-300.0 if j < 500 else j * 0.01)
    want, big = plain(q, pages, batch, vd, 1.0, 0, None, None)
    for parts in (1, 2, 5, 8):
        out = torch.empty(3, H, vd, dtype=torch.bfloat16, device=DEV)
        PG.attention_latent(q, pages, vd, batch, 0, 1.0, 0, None, None, out, parts)
        assert bool(((out.double() - want).abs() <= 2.0 ** -7 * (big + want.abs()) + 2e-3 * big).all())     # scores of 200: 1e-3 of float32 rounding


def test_a_page_that_is_not_there():
    from prelude_b200.ops import paged_general as PG
    q, pages, batch = make([300, 200], 16, 576, 512, 16, seed=6)
    batch.block_tables[0][0, 4] = -1
    want, big = plain(q, pages, batch, 512, 0.05, 0, None, None)
    for parts in (1, 4):
        out = torch.empty(2, 16, 512, dtype=torch.bfloat16, device=DEV)
        PG.attention_latent(q, pages, 512, batch, 0, 0.05, 0, None, None, out, parts)
        assert agrees(out, want, big)
    assert int(batch.status) == 0
    batch.block_tables[0][0, 4] = pages.shape[0]                  # a page outside the pool: reported, and left out
    PG.attention_latent(q, pages, 512, batch, 0, 0.05, 0, None, None, out)
    assert agrees(out, want, big) and int(batch.status) == 6


def test_other_calls_keep_the_general_kernel():
    from prelude_b200.ops import paged_general as PG
    q, pages, batch = make([100], 16, 576, 512, 16)
    assert not PG.latent_takes(q, pages, pages, 512, batch, 0, None, None)
    assert not PG.latent_takes(q, pages, None, 512, batch, 4, None, None)
    assert not PG.latent_takes(q, pages, None, 512, batch, 0, 64, None)
    assert not PG.latent_takes(q, pages, None, 512, batch, 0, None, 30.0)
    assert not PG.latent_takes(q.float(), pages, None, 512, batch, 0, None, None)
    assert not PG.latent_takes(q, pages, None, 480, batch, 0, None, None)
    assert not PG.latent_takes(q, pages, None, 512, batch, 0, None, None, PG.LATENT_MIN_ROWS_FEW - 1)
    batch.decode_only = False
    assert not PG.latent_takes(q, pages, None, 512, batch, 0, None, None)


@pytest.mark.parametrize("context,window,tokens", [(1023, None, 2), (1024, None, 2), (1500, 1000, 2), (1500, 1100, 2), (511, None, 8), (512, None, 8)])
def test_both_sides_of_the_rule_agree(context, window, tokens):
    # just below the rule's rows the general kernel takes the step, from there on this one: both within the weights' rounding
    from prelude_b200.ops import paged_general as PG
    q, pages, batch = make([context] + [300] * (tokens - 1), 16, 576, 512, 16, seed=8)
    pages[torch.isnan(pages)] = 0
    assert PG.latent_takes(q, pages, None, 512, batch, 0, None, None, min(context, window or context)) == (min(context, window or context) in (512, 1024, 1100))
    batch.cu_q, batch.max_q_len = torch.arange(tokens + 1, dtype=torch.int32, device=DEV), 1
    batch.workspace = lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device=DEV)
    want, big = plain(q, pages, batch, 512, 0.05, window or 0, None, None)
    assert agrees(PG.attention_general(q, pages, None, 512, batch, 0, 0.05, window, None), want, big)


def test_a_result_that_is_four_byte_aligned():
    # the general kernel takes it, as it did before there was another one
    from prelude_b200.ops import paged_general as PG
    H, vd = 16, 512
    q, pages, batch = make([1300, 1100, 40], H, 576, vd, 16, seed=9)
    pages[torch.isnan(pages)] = 0
    batch.cu_q, batch.max_q_len = torch.arange(4, dtype=torch.int32, device=DEV), 1
    batch.workspace = lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device=DEV)
    want, big = plain(q, pages, batch, vd, 0.05, 0, None, None)
    for offset in (2, 4, 8):
        out = torch.zeros(3 * H * vd + offset, dtype=torch.bfloat16, device=DEV)[offset:].view(3, H, vd)
        assert agrees(PG.attention_general(q, pages, None, vd, batch, 0, 0.05, None, None, out), want, big)
    assert int(batch.status) == 0

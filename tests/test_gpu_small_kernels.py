"""Kernels around the products, at the sizes where they change from one form to another, against the same in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# one rounding to the type (bfloat16: eight bits), and a few roundings of 6e-8 before it
UNIT = {torch.bfloat16: 2.0 ** -8 + 1e-6, torch.float32: 1.5e-6}


def _gen(seed=1):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [8, 12, 512, 516, 1536, 2048, 4104, 16384, 16392, 33000])
@pytest.mark.parametrize("rows", [1, 5])
def test_rmsnorm(dtype, width, rows):
    from prelude_b200.ops import kernels as K
    x = torch.randn(rows, width, generator=_gen(), device=DEV).to(dtype)
    w = torch.rand(width, generator=_gen(2), device=DEV) + 0.5
    y = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    got = K.rmsnorm(x, w, 1e-6).double()
    assert bool(((got - y).abs() <= UNIT[dtype] * y.abs() + 1e-12).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [64, 516, 2560, 8192, 8196, 9000])
@pytest.mark.parametrize("parts", [0, 1, 4, 6, None])
def test_final_norm_of_chosen_rows(dtype, width, parts):
    """parts 0: nothing joins; None: one output of the run's type; else float32 parts of a product."""
    from prelude_b200.ops import kernels as K
    res = torch.randn(9, width, generator=_gen(), device=DEV)
    w = torch.rand(width, generator=_gen(2), device=DEV) + 0.5
    rows = torch.tensor([8, 0, 3, 3, -1, 9], dtype=torch.int32, device=DEV)
    x, total = None, res.double()
    if parts is None:
        x = torch.randn(9, width, generator=_gen(3), device=DEV).to(dtype)
        total = total + x.double()
    elif parts:
        p = torch.randn(parts, 9, width, generator=_gen(3), device=DEV)
        x, total = K.PartialSums(p), total + p.double().sum(0)
    y = total / torch.sqrt((total ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    before = res.clone()
    got = K.gather_add_rmsnorm(x, res, rows, w, 1e-6, dtype).double()
    assert torch.equal(res, before)
    # the sum of up to seven terms is rounded at every step: 6e-8 of the terms, not of a sum that may cancel
    assert bool(((got[:4] - y[rows[:4].long()]).abs() <= UNIT[dtype] * y[rows[:4].long()].abs() + 4e-6).all())
    assert not got[4:].any()                               # no such row: zeros


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,inner,parts", [(2, 8192, 8), (2, 520, 1), (700, 8192, 8), (3, 4096, 1), (3, 4100, 1), (5, 96, 4), (3, 1026, 1)])
@pytest.mark.parametrize("gate_after", [False, True])
@pytest.mark.parametrize("sigmoid_gate", [False, True])
def test_gated_norm(dtype, T, inner, parts, gate_after, sigmoid_gate):
    from prelude_b200.ops import kernels as K
    y = torch.randn(T, inner, generator=_gen(), device=DEV)
    z = torch.randn(T, inner + 8, generator=_gen(2), device=DEV).to(dtype)[:, :inner]
    w = torch.rand(inner, generator=_gen(3), device=DEV) + 0.5
    g = torch.sigmoid(z.double()) * (1.0 if sigmoid_gate else z.double())
    v = y.double() if gate_after else y.double() * g
    v = v.view(T, parts, -1)
    v = (v / torch.sqrt((v ** 2).mean(-1, keepdim=True) + 1e-6)).view(T, inner) * w.double() * (g if gate_after else 1.0)
    got = K.gated_group_rmsnorm(y, z, w, parts, 1e-6, gate_after=gate_after, sigmoid_gate=sigmoid_gate).double()
    assert bool(((got - v).abs() <= UNIT[dtype] * v.abs() + 1e-12).all())


@pytest.mark.parametrize("requests", [1, 3])
@pytest.mark.parametrize("H,P,N,groups", [(8, 64, 128, 8), (4, 32, 64, 2), (2, 4, 5, 1), (2, 256, 16, 2), (3, 48, 128, 3), (2, 128, 300 - 44, 1)])
def test_state_space_step_of_single_tokens(requests, H, P, N, groups):
    """float32: a sum over N products, rounded N times at most and by far not all the same way."""
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.ops import kernels as K
    g = _gen(4)
    u = torch.randn(requests, H * P + 2 * groups * N, generator=g, device=DEV).bfloat16()
    dt = torch.randn(requests, H, generator=g, device=DEV).bfloat16()
    bias, a_log, skip = (torch.randn(H, generator=g, device=DEV) for _ in range(3))
    state = torch.randn(requests + 1, H, N, P, generator=g, device=DEV)
    batch = build_step_batch([StepItem(i, [0], 5) for i in range(requests)], {}, list(range(requests, 0, -1)), torch.device(DEV), 2, 100)
    S = state.double()[list(range(requests, 0, -1))]
    x, step = u.double()[:, :H * P].view(-1, H, P), torch.nn.functional.softplus(dt.double() + bias.double())
    B, C = (u.double()[:, H * P + k * groups * N:H * P + (k + 1) * groups * N].view(-1, groups, N).repeat_interleave(H // groups, 1) for k in (0, 1))
    decay = torch.exp(-torch.exp(a_log.double()) * step)
    S = decay[..., None, None] * S + (step.unsqueeze(-1) * B).unsqueeze(-1) * x.unsqueeze(2)
    want = ((S * C.unsqueeze(-1)).sum(2) + skip.double().view(1, H, 1) * x).flatten(1)
    before = state[0].clone()
    got = K.ssm_scan(u, dt, bias, a_log, skip, state, batch, groups)
    assert float((got.double() - want).norm() / want.norm()) < 1e-6
    assert float((state.double()[list(range(requests, 0, -1))] - S).norm() / S.norm()) < 1e-6
    assert torch.equal(state[0], before)                   # nobody's slot


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,d,rot,rank,dims", [(16, 128, 64, 512, 64), (32, 128, 64, 512, 32), (2, 32, 16, 64, 16), (5, 24, 8, 40, 8), (2, 16, 6, 24, 6),
                                               (40, 192, 64, 512, 64)])
@pytest.mark.parametrize("adjacent", [False, True])
@pytest.mark.parametrize("split", [True, False])
def test_queries_without_norm_beside_a_latent(dtype, H, d, rot, rank, dims, adjacent, split):
    """What is not turned is copied to the last bit; the normed latent is within its rounding; a turned element besides within what
    an angle's error, 2^-24 of the angle (2.4e-4 at position 3,999 and the fastest rate), its sine and cosine and three roundings
    leave of its pair's length."""
    from prelude_b200.ops import kernels as K
    g = _gen(6)
    T, pages, page = 7, 40, 4
    q = torch.randn(T, H * (d + rot) + 8, generator=g, device=DEV).to(dtype)[:, :H * (d + rot)]
    ckv = torch.randn(T, rank + rot, generator=g, device=DEV).to(dtype)
    w, rates = torch.rand(rank, generator=g, device=DEV) + 0.5, torch.rand(dims // 2, generator=g, device=DEV)
    pos = torch.tensor([0, 1, 2, 3, 4, 3999, 77], dtype=torch.int32, device=DEV)
    table = torch.full((3, 1000), -1, dtype=torch.int32, device=DEV)
    table[0, :2], table[2, 999], table[1, 19] = torch.tensor([5, 9], dtype=torch.int32, device=DEV), 30, 11
    rows = torch.tensor([0, 0, 0, 0, 0, 2, -1], dtype=torch.int32, device=DEV)
    k_pages = torch.zeros(pages, 1, page, rank + rot, dtype=dtype, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    cut = d if split else d + rot
    out, out2 = torch.zeros(T, H, cut, dtype=dtype, device=DEV), torch.zeros(T, H, rank + rot, dtype=dtype, device=DEV)
    K.qkv_prepare(q, ckv, None, n_heads=H, q_dim=d + rot, k_weight=w, k_norm_cols=rank, eps=1e-6, rates=rates, rot_dims=dims, adjacent=adjacent,
                  amplitude=1.25, q_rot_off=d, k_rot_off=rank, positions=pos, table_row=rows, block_table=table, q_out=out, q_split=cut,
                  q_out2=out2 if split else None, q2_off=rank, k_pages=k_pages, status=status)
    ang = pos.double().view(-1, 1, 1) * rates.double().view(1, 1, -1)
    c, s = ang.cos() * 1.25, ang.sin() * 1.25

    def turn(x):
        """The turned elements and what each may be off by, but for the result's rounding."""
        x, off = x.double().clone(), torch.zeros_like(x, dtype=torch.float64)
        first, second = (slice(0, dims, 2), slice(1, dims, 2)) if adjacent else (slice(0, dims // 2), slice(dims // 2, dims))
        a, b = x[..., first].clone(), x[..., second].clone()
        x[..., first], x[..., second] = a * c - b * s, b * c + a * s
        off[..., first] = off[..., second] = 1.25 * torch.hypot(a, b) * (ang * 2.0 ** -24 + 5 * 2.0 ** -23)
        return x, off

    live = rows >= 0
    heads = q.double().view(T, H, d + rot)
    turned, turned_off = turn(heads[..., d:])
    latent = ckv.double()[:, :rank]
    latent = latent / torch.sqrt((latent ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    key_turned, key_off = (x[:, 0] for x in turn(ckv[:, None, rank:]))
    got = (torch.cat([out, out2[..., rank:]], -1) if split else out).double()
    assert torch.equal(got[live][..., :d], heads[live][..., :d])
    assert bool(((got[..., d:] - turned).abs() <= UNIT[dtype] * turned.abs() + turned_off)[live].all())
    for t in range(T):
        if live[t]:
            have = k_pages[table[rows[t], int(pos[t]) // page].item(), 0, int(pos[t]) % page].double()
            assert bool(((have[:rank] - latent[t]).abs() <= UNIT[dtype] * latent[t].abs()).all())
            assert bool(((have[rank:] - key_turned[t]).abs() <= UNIT[dtype] * key_turned[t].abs() + key_off[t]).all())
    assert int(status) == 0 and not out[6].any()


@pytest.mark.parametrize("lens,H,G", [([700], 64, 4), ([700], 16, 4), ([65, 3, 64], 4, 2), ([2], 2, 1), ([1, 130], 6, 2), ([40], 64, 1)])
@pytest.mark.parametrize("vdim,dim", [(128, 64), (32, 16), (256, 128)])
@pytest.mark.parametrize("window", [None, 50])
def test_differential_attention_of_prompts(lens, H, G, vdim, dim, window):
    """Few tiles (their keys cut in two, put together inside a cluster) and many, against 64 bits: the weights enter the second
    product as bfloat16 (2^-9 each, of sums that the difference of two maps and the norm behind it may double), the result is
    rounded once more."""
    from prelude_b200.cache.manager import CacheManager
    from prelude_b200.config.spec import DiffAttentionSpec, QueryTemperatureSpec
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.ops import kernels as K
    from prelude_b200.ops.diff_attention import diff_attention
    from prelude_b200.parts.registry import KvPagesNeed
    g, T, dev = _gen(8), sum(lens), torch.device(DEV)
    spec = DiffAttentionSpec(hidden_size=64, num_heads=H, num_kv_heads=G, head_dim=dim, value_dim=vdim, softmax_scale=dim ** -0.5, lambda_init=0.5,
                             norm_eps=1e-6, query_temperature=QueryTemperatureSpec(coef=0.1, every=32), window=window)
    cache = CacheManager([KvPagesNeed(2 * G, dim, window, v_heads=G, v_head_dim=vdim)], 16, T // 16 + len(lens) + 1, len(lens), dev, torch.bfloat16)
    for r, n in enumerate(lens):
        cache.add_request(r)
        cache.grow(r, n)
    batch = build_step_batch([StepItem(r, [0] * n, 0) for r, n in enumerate(lens)], cache.block_tables(range(len(lens))),
                             [cache.slot_of(r) for r in range(len(lens))], dev, 2, 1 << 20)
    q, k, v, gate = (torch.randn(T, n, generator=g, device=DEV).bfloat16() for n in (H * 2 * dim, G * 2 * dim, G * vdim, H * vdim))
    mine = cache.layer_cache(0)
    K.kv_write_pages(k, v, mine.k_pages, mine.v_pages, batch.positions, batch.table_row_of_token, batch.block_tables[mine.group], batch.status)
    got = diff_attention(q, gate, mine.k_pages, mine.v_pages, batch, mine.group, spec, 0.3).double()
    at = 0
    for n in lens:
        i, j = torch.arange(n, device=DEV).view(-1, 1), torch.arange(n, device=DEV).view(1, -1)
        hidden = (j > i) | ((i - j >= window) if window else (j > i))
        tau = (1 + 0.1 * torch.log((torch.arange(1, n + 1, device=DEV) // 32 + 1).double())).view(1, n, 1)
        qq, kk = q[at:at + n].double().view(n, H, 2, dim), k[at:at + n].double().view(n, G, 2, dim).repeat_interleave(H // G, 1)
        vv = v[at:at + n].double().view(n, G, vdim).repeat_interleave(H // G, 1)
        maps = [torch.einsum("hij,jhe->ihe", torch.softmax((torch.einsum("ihd,jhd->hij", qq[:, :, c], kk[:, :, c]) * dim ** -0.5 * tau).masked_fill(hidden, -1e300), -1), vv)
                for c in (0, 1)]
        o = maps[0] - 0.3 * maps[1]
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * 0.5 * torch.sigmoid(gate[at:at + n].double().view(n, H, vdim))
        assert float((got[at:at + n] - o).norm() / o.norm()) < 6e-3
        at += n
    assert int(batch.status) == 0


@pytest.mark.parametrize("counts", [[1], [0, 31, 32, 33, 0], [255, 256, 257, 64, 0, 300, 1], [0, 0, 130], [520, 16, 200] * 5])
@pytest.mark.parametrize("K,N,act", [(64, 64, "silu"), (72, 136, "silu"), (200, 200, "clamped"), (328, 128, "silu"),
                                     (64, 128, "none"), (136, 264, "relu2"), (520, 328, "none")])
@pytest.mark.parametrize("max_pairs", [0, 3])
def test_products_of_routed_experts_on_paired_blocks(counts, K, N, act, max_pairs):
    """Experts with no rows, one, a step of columns more or less, and more than a tile, against 64 bits.  A float32 sum of products
    is within 2^-20 of the sum of their magnitudes, the result rounded once (2^-8 with the last bit of the exponential;
    2^-23 where it is float32)."""
    from prelude_b200.ops import kernels as K_
    from prelude_b200.ops.linear import tc_status
    g, E, T = _gen(21), len(counts), sum(counts)
    gated = act in ("silu", "clamped")
    if E * (2 * N if gated else N) < 128:
        pytest.skip("fewer rows than a block's")
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32, device=DEV) for e, n in enumerate(counts)])[torch.randperm(T, generator=g, device=DEV)].view(T, 1).contiguous()
    x = torch.randn(T, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, 2 * N if gated else N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    plan, status = K_.moe_sort(ids, E, 256), tc_status(torch.device(DEV))
    code = {"silu": K_.ACT_NONE, "none": K_.ACT_NONE, "clamped": K_.ACT_CLAMPED, "relu2": K_.ACT_RELU2}[act]
    rows = K_.moe_gather_rows(x, plan, 1)
    outs = [(K_.moe_gemm_grouped(rows, w, plan, gated, status, None, max_pairs, act=code, limit=0.8, alpha=1.7), 2.0 ** -8),
            (K_.moe_gemm_pair(rows, w, plan, gated, status, max_pairs, act=code, limit=0.8, alpha=1.7), 2.0 ** -8)]
    if not gated:
        outs.append((K_.moe_gemm_grouped(rows, w, plan, False, status, torch.float32, max_pairs, act=code), 2.0 ** -23))
    wd, xd, e = w.double(), x.double(), ids.view(-1).long()
    sums = torch.empty(T, w.shape[1], dtype=torch.float64, device=DEV)
    mags = torch.empty_like(sums)
    for i in range(E):
        sums[e == i], mags[e == i] = xd[e == i] @ wd[i].T, xd[e == i].abs() @ wd[i].abs().T
    err = mags * 2.0 ** -20
    if gated:
        a, b, ea, eb = sums[:, :N], sums[:, N:], err[:, :N], err[:, N:]
        if act == "clamped":
            a, b = a.clamp(max=0.8), b.clamp(-0.8, 0.8)
            want, slope, rest = a * torch.sigmoid(1.7 * a) * (b + 1), 1.2 * (b + 1).abs(), (a * torch.sigmoid(1.7 * a)).abs()
        else:
            want, slope, rest = a * torch.sigmoid(a) * b, 1.2 * b.abs(), (a * torch.sigmoid(a)).abs()
        bound = ea * slope + eb * rest
    elif act == "relu2":
        want, bound = sums.clamp(min=0) ** 2, 2 * err * (sums.abs() + err)
    else:
        want, bound = sums, err
    for out, unit in outs:
        assert ((out[plan.place_of.view(-1).long()].double() - want).abs() <= bound + want.abs() * unit + 1e-30).all()
    assert int(status) == 0


@pytest.mark.parametrize("width", [1, 255, 256, 257, 2047, 2048, 2049, 3000, 4096, 4097, 8192, 32000, 151936])
def test_argmax_of_rows_that_hold_minus_infinity(width):
    """Both loops over a chunk, eight loads at a time and the rest: a row of -inf alone gives its first index, one number among
    -inf wins wherever it stands, NaN never does (a row of NaN gives 0)."""
    from prelude_b200.ops import kernels as K
    places = sorted({0, width // 3, width // 2, width - 1})
    rows = torch.full((3 + len(places), width), float("-inf"), device=DEV)
    rows[1] = float("nan")
    rows[2, :(width + 1) // 2] = float("nan")               # then -inf, where there is more than one
    for r, at in enumerate(places):
        rows[3 + r, at] = -3.0e38
    got = K.argmax(rows).tolist()
    assert got == [0, 0, (width + 1) // 2 if width > 1 else 0] + places
    zero = torch.zeros(len(got), device=DEV)
    n = torch.zeros(len(got), dtype=torch.int64, device=DEV)
    assert K.sample(rows, zero, n, n).tolist() == got


@pytest.mark.parametrize("act", ["silu", "clamped"])
def test_gates_of_experts_with_few_rows_keep_32_bits(act):
    """Sums that 32 bits hold exactly (a gate: 21 bits of two products): what is left of a gate's error before its rounding to
    bfloat16 is the exponential's (two units in the last place at most) and three roundings, 4 x 2^-23 together.  Exponents from 20 to
    80, where the power of a rounded product is off by up to 40 units, and some of 200,000 results land on the wrong side."""
    from prelude_b200.ops import kernels as K
    from prelude_b200.ops.linear import tc_status
    g, counts, N = _gen(31), [191, 64, 130], 512
    T = sum(counts)
    ids = torch.repeat_interleave(torch.arange(3, device=DEV), torch.tensor(counts, device=DEV)).int().view(T, 1)
    x = torch.zeros(T, 64, device=DEV, dtype=torch.bfloat16)
    x[:, 0], x[:, 1] = -(20 if act == "silu" else 10) * (1 + torch.rand(T, generator=g, device=DEV)), 1
    x[:, 2] = torch.randint(0, 64, (T,), generator=g, device=DEV) / 256
    w = torch.zeros(3, 2 * N, 64, device=DEV, dtype=torch.bfloat16)
    w[:, :N, 0], w[:, N:, 1] = 1 + torch.rand(3, N, generator=g, device=DEV), 1
    w[:, :N, 2] = torch.randint(0, 64, (3, N), generator=g, device=DEV) / 64
    plan = K.moe_sort(ids, 3, 256)
    status = tc_status(torch.device(DEV))
    out = K.moe_gemm_grouped(K.moe_gather_rows(x, plan, 1), w, plan, True, status, None, 0, act=K.ACT_NONE if act == "silu" else K.ACT_CLAMPED,
                             limit=9.0, alpha=2.0)
    xd, wd = x.double(), w.double()[ids.view(-1).long()]
    z = xd[:, :1] * wd[:, :N, 0] + xd[:, 2:3] * wd[:, :N, 2]
    want = z * torch.sigmoid(z) if act == "silu" else 2 * z * torch.sigmoid(2 * z)
    half_unit = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(1e-300))) - 8)
    err = (out[plan.place_of.view(-1).long()].double() - want).abs()
    assert bool((err <= half_unit + want.abs() * 4 * 2.0 ** -23).all()) and int(status) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("adjacent", [False, True])
@pytest.mark.parametrize("H,d,dims", [(16, 128, 128), (64, 64, 64), (2, 32, 16)])
def test_queries_turned_where_they_lie(dtype, adjacent, H, d, dims):
    """``q_out`` the memory of ``q_in``: the same numbers as into memory of its own, but for the last bit (two kernels; a
    difference of two products of numbers below 6 may be off by 6 x 2^-23 in either)."""
    from prelude_b200.ops import kernels as K
    g, T = _gen(9), 300
    q = torch.randn(T, H * d, generator=g, device=DEV).to(dtype)
    rates = torch.rand(dims // 2, generator=g, device=DEV)
    pos, rows = torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)

    def turn(x, out):
        return K.qkv_prepare(x, None, None, n_heads=H, q_dim=d, rates=rates, rot_dims=dims, adjacent=adjacent, amplitude=1.0, positions=pos,
                             table_row=rows, q_out=out).clone()

    want = turn(q, torch.empty_like(q))
    for _ in range(3):
        mine = q.clone()
        got = turn(mine, mine)
        assert bool(((got.double() - want.double()).abs() <= 2 * UNIT[dtype] * want.double().abs() + 2 * 6 * 2.0 ** -23).all())


def test_gated_norm_of_more_parts_than_32_bits_count():
    # 2^31 parts of four: past what the kernel of a warp a part counts, and still taken
    from prelude_b200.ops import kernels as K
    if torch.cuda.mem_get_info()[0] < 90 << 30:
        pytest.skip("needs 70 GB")
    T, inner = 1 << 30, 8
    y = torch.zeros(T, inner, device=DEV)
    z = torch.zeros(T, inner, dtype=torch.bfloat16, device=DEV)
    w = torch.rand(inner, device=DEV) + 0.5
    where = [slice(0, 999), slice((1 << 29) - 500, (1 << 29) + 499), slice(T - 999, T)]
    for s in where:
        y[s], z[s] = torch.randn(999, inner, device=DEV), torch.randn(999, inner, device=DEV).bfloat16()
    got = K.gated_group_rmsnorm(y, z, w, 2, 1e-6)
    for s in where:
        v = (y[s].double() * torch.nn.functional.silu(z[s].double())).view(-1, 2, 4)
        want = (v * (v.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt()).view(-1, inner) * w.double()
        assert bool(((got[s].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())        # rounded to bfloat16 once


def _every_bfloat16():
    return torch.arange(1 << 16, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)


@pytest.mark.parametrize("form", ["gated", "columns", "sigmoid"])
def test_activations_give_the_same_bits_in_both_forms(form):
    # a row of eight elements an access and an element an access, which an odd address takes; every gate there is
    from prelude_b200.ops import kernels as K
    g, u = _every_bfloat16().view(64, 1024), torch.randn(64, 1024, generator=_gen(), device=DEV).bfloat16()

    def made(offset):
        if form == "gated":
            x = torch.empty(64 * 2048 + offset, dtype=torch.bfloat16, device=DEV)[offset:].view(64, 2048)
            x[:, :1024], x[:, 1024:] = g, u
            return K.silu_mul(x)
        x = torch.empty(64 * 1024 + offset, dtype=torch.bfloat16, device=DEV)[offset:].view(64, 1024)
        x.copy_(u if form == "sigmoid" else g)
        if form == "sigmoid":
            K.sigmoid_gate_(x, g)
        else:
            K.check(K._l.library().pb_silu_cols(x.data_ptr(), x.stride(0), K.dtype_code(x.dtype), 64, 1024, K._stream()), "silu_cols")
        return x
    a, b = made(0), made(1)
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(), b.nan_to_num())


@pytest.mark.parametrize("rank", [8, 16, 24, 32, 40, 64])
@pytest.mark.parametrize("T,channels", [(64, 128), (65, 129), (79, 1000), (2048, 40), (4100, 1024), (700, 2900)])
def test_channel_decays_by_rows_give_the_same_bits(rank, T, channels):
    # every number of tokens a block takes, against the kernel of eight tokens a block, which a matrix at an odd address goes to
    from prelude_b200.ops import kernels as K
    g = _gen(rank)
    x1 = torch.randn(T, rank + 8, generator=g, device=DEV).bfloat16()[:, 8:]
    room = torch.empty(channels * rank + 1, dtype=torch.bfloat16, device=DEV)
    w2 = (torch.randn(channels, rank, generator=g, device=DEV) / rank ** 0.5).bfloat16()
    odd = room[1:].view(channels, rank).copy_(w2)
    bias = torch.linspace(-60.0, 30.0, channels, device=DEV)
    got, want = K.channel_decay(x1, w2, bias, 16.0), K.channel_decay(x1, odd, bias, 16.0)
    assert torch.equal(got, want)
    z = x1.double() @ w2.double().T + bias.double()
    exact = torch.exp(torch.nn.functional.logsigmoid(z) / 16.0)
    # z from `rank` float32 products and sums of size below 60, a 16th of it in the exponent
    assert bool(((got.double() - exact).abs() <= (rank * 6e-8 * 8 + 60 * 6e-8 + 4e-7) * exact + 1e-12).all())

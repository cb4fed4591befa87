"""The router of prompt steps on the tensor cores, and the grouping of its choices, at the edges of their blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("E,groups,keep,top", [(8, 1, 1, 2), (32, 4, 2, 4), (33, 1, 1, 4), (64, 4, 2, 6), (65, 1, 1, 8), (256, 8, 4, 8)])
@pytest.mark.parametrize("T,K_", [(64, 32), (65, 96), (150, 4096), (2369, 1024)])
def test_router_of_a_prompt(T, K_, E, groups, keep, top):
    from prelude_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(T + E)
    x = torch.randn(T, K_ + 8, generator=g, device=DEV).bfloat16()[:, :K_]
    w = (torch.randn(E, K_, generator=g, device=DEV) * K_ ** -0.5).bfloat16()
    x[3, 5] = float("nan")                           # spoils its own row alone
    x[7] = 0.0                                       # every score ties: the smallest indices
    c = 0.1 * torch.randn(E, generator=g, device=DEV)
    c[: E // 2] = c[0]
    logits = torch.empty(T, E, device=DEV)
    args = (top, groups, keep, 2, True, c)
    ids, p = K.moe_route_tokens(x, w, *args, logits=logits)
    want = x.double() @ w.double().T
    ok = torch.arange(T, device=DEV) != 3
    # sums of sixteen cut to 2^-23 of the largest product (2^-24 in the root mean square); a warp adds them in twos, K / 512 of these, and the warps' sums
    # are added in 64 bits: that many sums rounded by 2^-25 of themselves, a warp's early ones of less
    assert float((logits[ok].double() - want[ok]).norm() / want[ok].norm()) < 2.0 ** -25 * (4 + 1 + (K_ / 512 + 1) / 2 + 1) ** 0.5
    assert bool(logits[3].isnan().all())
    ids2, p2 = K.moe_route(logits, *args)            # the choice is that of the logits alone
    assert torch.equal(ids, ids2) and torch.equal(p[ok], p2[ok])
    assert K.moe_route_tokens_takes(x, w) == (K_ >= 128 and (E > 8 or T <= 2368))


@pytest.mark.parametrize("K_", [128, 256, 512, 768, 1024, 4096])
def test_logits_are_no_less_exact_than_those_of_fewer_rows(K_):
    from prelude_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(K_)
    x, w = torch.randn(4096, K_, generator=g, device=DEV).bfloat16(), (torch.randn(64, K_, generator=g, device=DEV) * K_ ** -0.5).bfloat16()
    assert K.moe_route_tokens_takes(x, w)
    logits, want = torch.empty(4096, 64, device=DEV), x.double() @ w.double().T
    K.moe_route_tokens(x, w, 4, 1, 1, 1, False, logits=logits)
    assert float((logits.double() - want).norm()) <= float((K.router_logits(x, w).double() - want).norm())


def test_choices_by_a_plain_sort():
    """Largest score, then smallest index: with ties, signed zeros, infinities and NaN among the scores."""
    from prelude_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(3)
    z = torch.randint(-2, 3, (300, 96), generator=g, device=DEV).float()
    z[0, :] = torch.where(torch.arange(96, device=DEV) % 2 == 0, -0.0, 0.0)
    z[1, 5], z[1, 6], z[2, 9] = float("inf"), -float("inf"), float("nan")
    ids, _ = K.moe_route(z, 6, 1, 1, 1, False, softmax_chosen=True)
    for t in range(300):
        order = sorted((e for e in range(96) if z[t, e] > -float("inf")), key=lambda e: (-float(z[t, e]) + 0.0, e))
        assert ids[t].tolist() == order[:6]


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (7, 6, 64), (341, 6, 64), (342, 6, 64), (2048, 6, 64), (1000, 8, 1024), (12000, 6, 40), (64, 2, 4), (129, 1, 8),
                                      (256, 2, 9), (513, 1, 300), (2047, 1, 5), (2048, 1, 5)])
def test_grouping(T, top, E):
    from prelude_b200.ops import kernels as K
    ids = torch.randint(0, E, (T, top), generator=torch.Generator(device=DEV).manual_seed(T), device=DEV).int()
    plan = K.moe_sort(ids, E, 256)
    flat, order, n = ids.flatten().long(), plan.order.long(), T * top
    counts = torch.bincount(flat, minlength=E)
    assert torch.equal(order.sort().values, torch.arange(n, device=DEV)) and bool((flat[order].diff() >= 0).all())
    assert torch.equal(plan.place_of.long()[order], torch.arange(n, device=DEV))
    assert torch.equal(plan.offsets.long(), torch.cat([counts.new_zeros(1), counts.cumsum(0)]))
    tiles = [(e, int(plan.offsets[e]) + k) for e in range(E) for k in range(0, int(counts[e]), 256)]
    got = list(zip(plan.tile_expert.tolist(), plan.tile_row0.tolist()))
    assert got[:len(tiles)] == tiles and all(e == -1 for e, _ in got[len(tiles):])


@pytest.mark.parametrize("T,top,width,y32", [(5, 3, 64, True), (9, 6, 4096, False), (70, 8, 520, False), (70, 9, 520, True), (3, 17, 100, False),
                                             (300, 1, 2880, False), (40, 2, 512, False), (5, 1, 512, True), (33, 4, 2048, False), (7, 5, 2048, False)])
def test_weighted_sum(T, top, width, y32):
    from prelude_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(top)
    y = torch.randn(T * top, width, generator=g, device=DEV)
    y = y if y32 else y.bfloat16()
    w = torch.rand(T, top, generator=g, device=DEV)
    place = torch.randperm(T * top, generator=g, device=DEV).int()
    got = K.PendingExperts(y, place, w, None, torch.bfloat16).resolve().double()
    want = (y[place.long()].double().view(T, top, width) * w.double().unsqueeze(-1)).sum(1)
    # `top` roundings of the running sum, whose size the terms bound, and one to bfloat16
    size = (y[place.long()].double().abs().view(T, top, width) * w.double().unsqueeze(-1)).sum(1)
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + top * 2.0 ** -24 * size).all())


@pytest.mark.parametrize("T,E,K_", [(64, 64, 4096), (100, 8, 1024), (64, 200, 2048)])
def test_both_routers_choose_alike_away_from_ties(T, E, K_):
    """A token's logits come from another order of sums from 64 rows on: they differ by roundings, and its experts only where two tie within them."""
    from prelude_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(E)
    x, w = torch.randn(T, K_, generator=g, device=DEV).bfloat16(), (torch.randn(E, K_, generator=g, device=DEV) * K_ ** -0.5).bfloat16()
    logits, args = torch.empty(T, E, device=DEV), (4, 1, 1, 1, False)
    ids, _ = K.moe_route_tokens(x, w, *args, softmax_chosen=True, logits=logits)
    few = K.router_logits(x, w)
    ids_few, _ = K.moe_route(few, *args, softmax_chosen=True)
    # K / 32 sums a lane and five between lanes; sums of sixteen cut in sixteen places, K / 512 pairs of them and one rounding at the end
    most = 2.0 ** -24 * ((K_ / 32 + 5) + (32 + K_ / 512 + 2)) * (x.double().abs() @ w.double().abs().T)
    assert bool(((logits.double() - few.double()).abs() <= most).all())
    order = few.double().sort(1, descending=True).values[:, :5]
    apart = (order[:, :4] - order[:, 1:]).min(1).values > 2 * most.max()
    assert int(apart.sum()) > T // 2 and torch.equal(ids[apart], ids_few[apart])

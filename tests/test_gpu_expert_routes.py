"""Which products a step's routed experts run on, on both sides of the rule's ends, and that the whole feed-forward is the same there."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_the_rule():
    from prelude_b200.parts.moe import grouped_pays
    for width, ff, mats in ((4096, 2048, 3), (4096, 2048, 2), (2048, 2048, 2), (2048, 768, 3), (1024, 512, 2)):
        size = mats * width * ff * 2
        for experts, top in ((8, 2), (8, 4), (16, 6), (32, 4), (64, 8), (4, 4)):
            takes = [grouped_pays(t, top, experts, size) for t in range(1, 65)]
            assert not takes[0]                      # one token hits every expert once: nothing is read twice
            assert takes == sorted(takes)            # and from some token on it pays
    assert not grouped_pays(2, 4, 8, 2 * 4096 * 2048 * 2) and not grouped_pays(8, 4, 32, 2 * 2048 * 2048 * 2) and grouped_pays(24, 4, 32, 2 * 2048 * 2048 * 2)


def made(g, activation, width, ff, experts, top):
    from prelude_b200.config.spec import RoutedExpertsSpec
    from prelude_b200.parts import model as _registers_the_parts  # noqa: F401
    from prelude_b200.parts.registry import RunContext, make_part
    w = {"ff.router": torch.randn(experts, width, generator=g, device=DEV) * width ** -0.5}
    for e in range(experts):
        if activation == "silu_gated":
            w[f"ff.e{e}.gate"] = torch.randn(ff, width, generator=g, device=DEV) * width ** -0.5
        w[f"ff.e{e}.up"] = torch.randn(ff, width, generator=g, device=DEV) * width ** -0.5
        w[f"ff.e{e}.down"] = torch.randn(width, ff, generator=g, device=DEV) * ff ** -0.5
    w = {n: t.bfloat16() for n, t in w.items()}
    part = make_part("feed_forward", RoutedExpertsSpec(width, ff, experts, top, activation=activation), "ff")
    part.load(lambda n: w[n], RunContext(torch.device(DEV), torch.bfloat16))
    return part, w


def watched(monkeypatch):
    from prelude_b200.ops import kernels as K
    taken = []
    for name in ("moe_gemv", "moe_gemm_grouped", "moe_gemm"):
        monkeypatch.setattr(K, name, lambda *a, _f=getattr(K, name), _n=name, **k: (taken.append(_n), _f(*a, **k))[1])
    return taken


@pytest.mark.parametrize("activation", ["silu_gated", "relu2"])
@pytest.mark.parametrize("width,ff,experts,top,below,above", [(2048, 768, 16, 2, {"silu_gated": 21, "relu2": 25}, {"silu_gated": 22, "relu2": 26}),
                                                              (4096, 2048, 8, 2, {"silu_gated": 7, "relu2": 8}, {"silu_gated": 8, "relu2": 9}),
                                                              (1024, 512, 8, 2, {"silu_gated": 24, "relu2": 24}, {"silu_gated": 25, "relu2": 25})])
def test_both_sides(activation, width, ff, experts, top, below, above, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(width + experts)
    gated = activation == "silu_gated"
    part, w = made(g, activation, width, ff, experts, top)
    taken = watched(monkeypatch)
    for T, kernel in ((below[activation], "moe_gemv"), (above[activation], "moe_gemm_grouped")):
        x = torch.randn(T, width, generator=g, device=DEV).bfloat16()
        ids, p = part.route(x)
        taken.clear()
        y = part.forward(x)
        assert set(taken) == {kernel}
        h, want = x.double(), torch.zeros(T, width, dtype=torch.float64, device=DEV)
        for e in range(experts):
            m = {n: w[f"ff.e{e}.{n}"].double() for n in (("gate", "up", "down") if gated else ("up", "down"))}
            a = torch.nn.functional.silu(h @ m["gate"].T) * (h @ m["up"].T) if gated else torch.relu(h @ m["up"].T) ** 2
            want += ((ids == e) * p.double()).sum(1, keepdim=True) * (a @ m["down"].T)
        # the activation and the result rounded to bfloat16: 1.7e-3 each in the 2-norm
        assert float((y.double() - want).norm() / want.norm()) < 4e-3


@pytest.mark.parametrize("rows,kernel", [("1", "moe_gemm_grouped"), ("1000000", "moe_gemv")])
def test_rows_that_the_caller_sets_go_before_the_rule(rows, kernel, monkeypatch):
    from prelude_b200.parts import moe
    part, _ = made(torch.Generator(device=DEV).manual_seed(4), "silu_gated", 2048, 768, 16, 2)
    taken = watched(monkeypatch)
    monkeypatch.setattr(moe, "MOE_GROUPED_ROWS_SET", rows)
    for T in (8, 24, 40):                            # one row an expert and more: the rule alone takes the last two
        part.forward(torch.randn(T, 2048, device=DEV).bfloat16())
        assert set(taken) == {kernel}
        taken.clear()

"""Which products a step's routed experts run on, on both sides of the rule's ends, and that the whole feed-forward is the same there."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_the_rule():
    from prelude_b200.parts.moe import grouped_min_rows
    assert grouped_min_rows(4096 * 2048, True) == grouped_min_rows(2048 * 768, True) == 1.5
    assert (grouped_min_rows(4096 * 2048, False), grouped_min_rows(2048 * 2048, False)) == (0.375, 1.0)
    assert grouped_min_rows(1024 * 512, True) == grouped_min_rows(1024 * 512, False) == float("inf")


@pytest.mark.parametrize("activation", ["silu_gated", "relu2"])
@pytest.mark.parametrize("width,ff,experts,top,below,above", [(2048, 768, 16, 2, {"silu_gated": 11, "relu2": 7}, {"silu_gated": 12, "relu2": 8}),
                                                              (4096, 2048, 8, 2, {"silu_gated": 5, "relu2": 1}, {"silu_gated": 6, "relu2": 2}),
                                                              (1024, 512, 8, 2, {"silu_gated": 24, "relu2": 24}, {"silu_gated": 25, "relu2": 25})])
def test_both_sides(activation, width, ff, experts, top, below, above, monkeypatch):
    from prelude_b200.config.spec import RoutedExpertsSpec
    from prelude_b200.ops import kernels as K
    from prelude_b200.parts import model as _registers_the_parts  # noqa: F401
    from prelude_b200.parts.registry import RunContext, make_part
    g = torch.Generator(device=DEV).manual_seed(width + experts)
    gated = activation == "silu_gated"
    w = {"ff.router": torch.randn(experts, width, generator=g, device=DEV) * width ** -0.5}
    for e in range(experts):
        if gated:
            w[f"ff.e{e}.gate"] = torch.randn(ff, width, generator=g, device=DEV) * width ** -0.5
        w[f"ff.e{e}.up"] = torch.randn(ff, width, generator=g, device=DEV) * width ** -0.5
        w[f"ff.e{e}.down"] = torch.randn(width, ff, generator=g, device=DEV) * ff ** -0.5
    w = {n: t.bfloat16() for n, t in w.items()}
    part = make_part("feed_forward", RoutedExpertsSpec(width, ff, experts, top, activation=activation), "ff")
    part.load(lambda n: w[n], RunContext(torch.device(DEV), torch.bfloat16))
    taken = []
    for name in ("moe_gemv", "moe_gemm_grouped"):
        monkeypatch.setattr(K, name, lambda *a, _f=getattr(K, name), _n=name, **k: (taken.append(_n), _f(*a, **k))[1])
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

"""The router's kernels take rows of the router matrix's width and type alone: others are refused before anything is launched."""
import pytest
import torch

from prelude_b200.config.spec import RoutedExpertsSpec
from prelude_b200.ops import kernels as K
from prelude_b200.parts import model as _registers_the_parts  # noqa: F401
from prelude_b200.parts.registry import RunContext, make_part

WIDTH, E = 2048, 8


@pytest.fixture
def launched(monkeypatch):
    """The library's questions are answered by itself (they need no GPU), its launches only written down; host tensors pass for the GPU's."""
    real, names = K._l.library(), []

    class Library:
        def __getattr__(self, name):
            if name.endswith(("_supported", "_takes")):
                return getattr(real, name)
            return lambda *a: names.append(name) or 0

    def need(t, name, dtype=None, contiguous=True):
        if (dtype is not None and t.dtype != dtype) or (contiguous and not t.is_contiguous()):
            raise K.KernelLibraryError(f"{name}: {t.dtype}, not {dtype}, or not contiguous")

    monkeypatch.setattr(K._l, "library", lambda: Library())
    monkeypatch.setattr(K, "_need", need)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    return names


@pytest.mark.parametrize("route", ["moe_route_few", "moe_route_tokens", "router_logits"])
def test_a_router_refuses_rows_of_another_width_or_type(route, launched):
    w, args = torch.zeros(E, WIDTH, dtype=torch.bfloat16), () if route == "router_logits" else (2, 1, 1, 1, False)
    for width, dtype in ((WIDTH + 32, torch.bfloat16), (WIDTH - 32, torch.bfloat16), (WIDTH, torch.float32)):
        x = torch.zeros(64, width, dtype=dtype)
        assert not K.moe_route_few_takes(x, w) and not K.moe_route_tokens_takes(x, w)
        with pytest.raises(K.KernelLibraryError):
            getattr(K, route)(x, w, *args)
    assert launched == []
    getattr(K, route)(torch.zeros(64, WIDTH, dtype=torch.bfloat16), w, *args)
    assert launched == ["pb_" + route]


def test_the_tensor_cores_router_refuses_float32(launched):
    with pytest.raises(K.KernelLibraryError):
        K.moe_route_tokens(torch.zeros(64, WIDTH), torch.zeros(E, WIDTH), 2, 1, 1, 1, False)
    assert launched == []


@pytest.mark.parametrize("rows", [8, 40, 64])
@pytest.mark.parametrize("width", [WIDTH - 32, WIDTH + 32])
def test_routed_experts_refuse_rows_of_another_width(rows, width, launched):
    part = make_part("feed_forward", RoutedExpertsSpec(WIDTH, 32, E, 2), "ff")
    part.load(lambda n: torch.zeros([t for t in part.tensors().items() if t[0] == n][0][1].shape), RunContext(torch.device("cpu"), torch.bfloat16))
    x = torch.zeros(rows, width, dtype=torch.bfloat16)
    for call in (part.route, part.forward):
        with pytest.raises(K.KernelLibraryError):
            call(x)
    assert launched == []
    part.route(torch.zeros(rows, WIDTH, dtype=torch.bfloat16))
    assert launched[0] == {8: "pb_moe_route_few", 40: "pb_router_logits", 64: "pb_moe_route_tokens"}[rows]


# one wave of blocks: long rows, or products enough; more waves: many experts with long rows, or a whole block's worth of experts
@pytest.mark.parametrize("tokens,experts,width,taken", [
    (63, 64, 4096, False), (64, 2, 2048, True), (64, 8, 1024, False), (1600, 16, 1024, True), (800, 16, 512, False), (1600, 24, 512, True), (64, 65, 128, True), (64, 64, 96, False),
    (2368, 8, 4096, True), (2369, 8, 4096, False), (2369, 9, 4096, True), (16384, 16, 1024, False), (16384, 32, 1024, True), (16384, 64, 128, True)])
def test_where_the_tensor_cores_router_pays(tokens, experts, width, taken):
    if torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the waves are those of 148 multiprocessors")
    assert bool(K._l.library().pb_moe_route_tokens_supported(tokens, experts, width)) == taken

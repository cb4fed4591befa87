"""Which of the experts' kernels a step of few rows runs on: the rules alone, no GPU."""
import pytest
import torch

from prelude_b200.config.spec import RoutedExpertsSpec
from prelude_b200.parts import model as _registers_the_parts  # noqa: F401
from prelude_b200.parts.registry import make_part


# with matrices whose rows go through a ring, long and short ones, and with rows too short for it; few experts, whose line is the old one
@pytest.mark.parametrize("width,ff,experts,top,tokens,grouped", [
    (4096, 2048, 64, 6, 16, False), (4096, 2048, 64, 6, 32, False), (4096, 2048, 128, 8, 64, False), (2048, 2048, 32, 4, 40, False), (1536, 1040, 64, 8, 48, False),
    (2048, 768, 64, 8, 23, False), (2048, 768, 64, 8, 24, True), (1024, 1024, 128, 8, 64, True), (2048, 768, 32, 8, 24, False),
    (4096, 512, 64, 8, 30, True), (4096, 2048, 16, 2, 12, False), (4096, 2048, 16, 4, 12, True), (4096, 2048, 8, 2, 7, False), (4096, 2048, 8, 2, 8, True)])
def test_sides_of_the_rules(width, ff, experts, top, tokens, grouped):
    part = make_part("feed_forward", RoutedExpertsSpec(width, ff, experts, top), "ff")
    part.w_gate_up, part.w_down = torch.empty(experts, 2 * ff, width, device="meta"), torch.empty(experts, width, ff, device="meta")
    assert part._grouped(torch.zeros(tokens, width, dtype=torch.bfloat16), True) == grouped

"""Which of the experts' kernels a step of few rows runs on: the rules alone, no GPU."""
import itertools

import pytest
import torch

from prelude_b200.config.spec import RoutedExpertsSpec
from prelude_b200.parts import model as _registers_the_parts  # noqa: F401
from prelude_b200.parts import moe
from prelude_b200.parts.registry import make_part


@pytest.mark.parametrize("tokens,top,experts", [(8, 1, 2), (9, 1, 2), (10, 1, 2), (10, 2, 3), (9, 3, 3)])
def test_experts_with_more_than_eight_tokens(tokens, top, experts):
    """Against every way in which the tokens may choose."""
    chosen = list(itertools.combinations(range(experts), top))
    n = sum(sum(0 in c for c in each) > 8 for each in itertools.product(chosen, repeat=tokens))      # expert 0 has more than eight
    assert moe.nine_or_more(tokens, top / experts) == pytest.approx(n / len(chosen) ** tokens)


# with matrices whose rows go through a ring, and with shorter ones
@pytest.mark.parametrize("width,ff,experts,top,tokens,grouped", [
    (4096, 2048, 64, 6, 16, False), (4096, 2048, 64, 6, 32, True), (4096, 2048, 128, 8, 20, False), (2048, 2048, 32, 4, 12, False), (2048, 2048, 32, 4, 32, True), (4096, 2048, 16, 2, 12, False), (4096, 2048, 16, 4, 12, True),
    (4096, 512, 64, 8, 30, True), (4096, 2048, 8, 2, 7, False), (4096, 2048, 8, 2, 8, True)])
def test_sides_of_the_rules(width, ff, experts, top, tokens, grouped):
    part = make_part("feed_forward", RoutedExpertsSpec(width, ff, experts, top), "ff")
    part.w_gate_up, part.w_down = torch.empty(experts, 2 * ff, width, device="meta"), torch.empty(experts, width, ff, device="meta")
    assert part._grouped(torch.zeros(tokens, width, dtype=torch.bfloat16), True) == grouped

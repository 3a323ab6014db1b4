"""Which of two kernels a step takes: the rules against steps that were timed both ways on a B200.

The lines are drawn from estimates that are within 10 % of a time, so only steps are asked for here whose two times are a
quarter and more apart."""

from __future__ import annotations

import pytest

from distie_b200.kernels.device import chunks_pay


@pytest.mark.parametrize("rule,key,value,heads,portions,tokens,walk,chunks", [
    # rule, sizes, heads, portions, tokens of each, us token by token, us in chunks
    ("delta", 16, 16, 40, 16, 155, 65.6, 247.9),
    ("delta", 32, 32, 28, 16, 155, 74.6, 210.0),
    ("delta", 64, 64, 40, 16, 155, 242.1, 398.6),
    ("delta", 64, 64, 40, 4, 158, 69.3, 114.9),
    ("delta", 128, 128, 12, 4, 64, 32.4, 49.0),
    ("delta", 128, 128, 12, 1, 2048, 507.0, 169.0),
    ("delta", 16, 16, 4, 1, 512, 83.0, 33.9),
    ("delta", 96, 96, 40, 1, 1024, 320.5, 196.4),
    ("ssd", 16, 16, 40, 16, 71, 27.8, 82.0),
    ("ssd", 32, 32, 28, 16, 72, 30.5, 65.9),
    ("ssd", 128, 128, 1, 1, 96, 20.2, 28.5),
    ("ssd", 128, 128, 12, 1, 2048, 372.0, 92.0),
    ("ssd", 128, 128, 40, 32, 64, 682.8, 314.7),
    ("gated", 16, 16, 40, 16, 71, 33.8, 82.0),
    ("gated", 32, 32, 12, 16, 80, 21.6, 36.4),
    ("ssd", 128, 128, 24, 4, 256, 180.6, 80.5),
])
def test_recurrences_run_in_chunks_where_that_is_faster(rule, key, value, heads, portions, tokens, walk, chunks):
    assert chunks_pay(rule, portions * tokens, portions, heads, key, value) == (chunks < walk)

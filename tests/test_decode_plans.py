"""Which split of the keys decode attention takes by head size, pairs of rows and kv heads, and the longest context."""

from __future__ import annotations

import pytest

from research_2_b200.kernels import ops


@pytest.fixture(autouse=True)
def sms(monkeypatch):
    monkeypatch.setattr(ops, "sm_count", lambda device="cuda:0": 148)


# head sizes above 64 have no half of a wide CTA that would be wide itself: narrow CTAs, sliced where the chip has room
@pytest.mark.parametrize("pairs,hd,context,plan", [
    (160, 80, 1024, (2, 4)), (160, 128, 1024, (1, 4)), (160, 128, 4096, (3, 4)), (192, 96, 4096, (3, 4)), (200, 128, 4096, (1, 4)), (200, 80, 4096, (2, 4)),
    (296, 80, 4096, (1, 4)), (297, 128, 4096, (1, 4)), (160, 80, 100, (1, 4)),
    (160, 64, 1024, (1, 8)), (160, 64, 4096, (3, 4)), (200, 64, 4096, (1, 8)), (296, 64, 4096, (1, 8)), (297, 64, 4096, (1, 4)),
])
def test_more_pairs_than_sms(pairs, hd, context, plan):
    assert ops.decode_plan(pairs, 1, hd, context) == plan


@pytest.mark.parametrize("pairs,hd,context,plan", [
    (8, 128, 600, (2, 8)), (8, 128, 640, (2, 8)), (8, 128, 768, (3, 8)), (8, 128, 1024, (4, 8)), (16, 80, 1024, (4, 8)), (17, 80, 1024, (2, 8)), (8, 96, 8192, (8, 8)), (148, 128, 8192, (1, 8)),
    (8, 64, 1024, (1, 16)), (8, 64, 4096, (4, 16)), (74, 64, 4096, (2, 16)),
])
def test_up_to_a_pair_an_sm(pairs, hd, context, plan):
    assert ops.decode_plan(1, pairs, hd, context) == plan

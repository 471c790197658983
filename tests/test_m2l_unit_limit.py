"""Pairs per M2L unit: a power of two in its range, an even share of the far
list over the resident threads, and never shorter for a longer list."""

from __future__ import annotations

import pytest

from jaccpot_b200.schedule import M2L_RESIDENT_THREADS as T, m2l_unit_limit


@pytest.mark.parametrize("mixed,share,most", [(False, 1, 512), (True, 2, 64)])
def test_limit_is_the_even_share_within_its_range(mixed, share, most):
    last = 8
    for pairs in [0, 1, 7 * T, 8 * T, 8 * T + 1, 16 * T * share, 16 * T * share + 1, 100 * T, 500 * T, 513 * T, 10**10]:
        got = m2l_unit_limit(pairs, mixed)
        assert 8 <= got <= most and got & (got - 1) == 0
        assert got == most or got * T * share >= pairs
        assert got == 8 or (got // 2) * T * share < pairs
        assert got >= last
        last = got

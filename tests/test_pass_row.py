"""The pre-pass takes a unit's row by a product with the rounded-up 2^32 / group where it holds that to be exact: held to the division here, at both
sides of multiples of the group up to the last unit that the rule admits."""
import pytest


def per_head(rows, group):
    """prepass.cuh pass_add"""
    if group > 1 and (rows * group + (1 << 20)) * group < 1 << 32:
        return ((1 << 32) + group - 1) // group
    return 0


@pytest.mark.parametrize("group", [2, 3, 4, 5, 6, 7, 8, 12, 17, 31, 33, 64, 100, 511, 1000, 2000])
def test_rows_by_a_product(group):
    m = per_head(1, group)
    most = (1 << 32) // group - (1 << 20)  # units of the largest sequence that the rule admits
    rows = max(0, most // group - 1)
    assert m and (rows == 0 or per_head(rows, group) == m)
    last = rows * group + (1 << 20) - 1  # (the last block's lanes look a few steps further)
    for r in {0, 1, 2, 1000, 65535, last // group // 2, last // group}:
        for u in (r * group, r * group + 1, r * group + group - 1):
            if u <= last:
                assert u * m >> 32 == u // group, u
    assert per_head(1 << 31, group) == 0 and per_head(5, 1) == 0

"""The kernels' division of a cell index by the row length (fast_div), on the host."""
import pytest


@pytest.mark.parametrize("d", [2, 3, 5, 16, 31, 100, 12345, 65537, 1 << 20, (1 << 30) + 7])
def test_fast_division_rule(d):
    """The multiplier and shift the kernels divide by (fast_div), on the host."""
    s = 1
    while (1 << s) < d:
        s += 1
    m = -(-(1 << (31 + s)) // d)
    assert m < 1 << 32
    for q in {0, 1, 2, (2 ** 31 - 1) // d // 2, (2 ** 31 - 1) // d}:
        for i in (q * d - 1, q * d, q * d + 1, 2 ** 31 - 1):
            if 0 <= i < 2 ** 31:
                assert ((i * m) >> 32) >> (s - 1) == i // d

"""The benchmark's byte model of a split product counts what the kernels read."""
from __future__ import annotations

import pytest


@pytest.mark.parametrize("P,Q", [(32, 64), (5, 8), (7, 9)])
def test_the_product_is_credited_with_each_distinct_spectra_value_once(P, Q):
    """Entry m of the subband of parity p on n frequencies equals entry n - m - p (mod n), along both axes, and a product
    reads the lower of the two: the distinct pairs over four subbands, three generators each."""
    import bench

    def lower(n, p):
        return len({min(m, (n - m - p) % n) for m in range(n)})

    distinct = 3 * sum(lower(P, px) * lower(Q, py) for px in (0, 1) for py in (0, 1))
    assert bench.matvec_bytes(100, P, Q, 16) == 16 * (2 * 100 + 16 * P * Q + distinct)

"""Counts of catalogs whose field labels interleave in space, so that leaves
break into runs of one or two points and query blocks hold many fields, against
the oracle's exhaustive counts (exact: integers, no tolerance)."""
import numpy as np
import pytest

from corruscant_b200 import _native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 5, 6, 15, 16, 17, 33, 120, 255])
@pytest.mark.parametrize("n", [40, 128, 700, 2500])
def test_random_labels(n, nf):
    """Numbers of fields at and next to those where the kernel changes its way,
    symmetric and crossed, in one pass and (KD_MAX_EDGES) in two."""
    rs = np.random.RandomState(1000 * n + nf)
    p, q = rs.rand(n, 3), rs.rand(n // 2 + 1, 3)
    f, g = (rs.randint(0, nf, len(x)).astype(np.int32) for x in (p, q))
    f[0] = g[0] = nf - 1
    ot = O.OracleTree(p, f, nf)
    t, tq = N.build_tree(p, f, nf), N.build_tree(q, g, nf)
    try:
        for radii in (np.linspace(0.02, 1.2, 9), np.linspace(0.01, 0.9, 66 if nf < 20 else 5)):
            auto = ot.brute_counts(p, f, nf, radii, nthreads=4)
            cross = ot.brute_counts(q, g, nf, radii, nthreads=4)
            for mode in (N.KD_MODE_MIXED, N.KD_MODE_FP64):
                assert np.array_equal(N.count_radii(t, t, radii, mode=mode), auto), mode
                assert np.array_equal(N.count_radii(t, tq, radii, mode=mode), cross), mode
                assert np.array_equal(N.count_points(t, q, g, nf, radii, mode=mode), cross), mode
            if nf < 20 and len(radii) <= 64:
                assert np.array_equal(N.count_radii_static(t, tq, radii), cross)
    finally:
        N.destroy(t)
        N.destroy(tq)

"""Counts at the sizes where the tile kernel's layouts end: runs, query blocks
and query tiles one short of, at and one past their limits, and windows of one
edge up to several passes, against the oracle's exhaustive counts (exact:
integers, no tolerance)."""
import numpy as np
import pytest

from corruscant_b200 import _native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MODES = (N.KD_MODE_MIXED, N.KD_MODE_FP64)


def _check(tp, tf, qp, qf, nf, radii):
    ot = O.OracleTree(tp, tf, nf)
    want = ot.brute_counts(qp, qf, nf, radii, nthreads=4)
    t, q = N.build_tree(tp, tf, nf), N.build_tree(qp, qf, nf)
    try:
        for mode in MODES:
            assert np.array_equal(N.count_radii(t, q, radii, mode=mode), want), mode
            auto = N.count_radii(q, q, radii, mode=mode)  # symmetric, runs cut at the blocks
            assert np.array_equal(auto, O.OracleTree(qp, qf, nf).brute_counts(
                qp, qf, nf, radii, nthreads=4)), mode
    finally:
        N.destroy(t)
        N.destroy(q)


@pytest.mark.parametrize("ne", [1, 2, 3, 4, 5, 9, 64])
@pytest.mark.parametrize("nt,nq", [(1, 1), (7, 15), (8, 16), (9, 17), (63, 127), (64, 128),
                                   (65, 129), (129, 31), (200, 257), (1000, 3)])
def test_sizes_and_window_widths(nt, nq, ne):
    rs = np.random.RandomState(1000 * nt + nq + ne)
    tp, qp = rs.rand(nt, 3), rs.rand(nq, 3)
    tf, qf = (tp[:, 0] * 3).astype(np.int32), (qp[:, 1] * 3).astype(np.int32)
    _check(tp, tf, qp, qf, 3, np.linspace(0.05, 1.6, ne))


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1e-6, 1.0), (1e-18, 0.0), (1e9, 3e11),
                                          (1e14, 0.0), (3e17, 1e18)])
def test_scales_and_on_edge_pairs(scale, offset):
    """Lattice points (pairs exactly on edges) and points with edges spread
    over six decades, at scales inside and outside FP32's range."""
    rs = np.random.RandomState(5)
    lat = rs.randint(0, 9, (700, 3)) / 8.0
    _check(lat * scale + offset, None, lat[:300] * scale + offset, None, 1,
           np.sqrt(np.array([1, 2, 3, 5, 9, 20, 70]) / 64.0) * scale)
    p = np.concatenate([rs.rand(600, 3), rs.rand(600, 3) * 1e-4])
    _check(p * scale + offset, None, p[::3] * scale + offset, None, 1,
           np.array([1e-6, 3e-5, 1e-4, 0.01, 0.3, 1.0, 50.0]) * scale)

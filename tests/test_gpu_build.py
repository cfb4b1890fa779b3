"""Trees at the sizes where the build's kernels change, node for node against
the oracle (bit for bit: no tolerance)."""
import numpy as np
import pytest

from corruscant_b200 import _native as N
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(p, f, nf):
    t = N.build_tree(p, f, nf)
    try:
        got, want = N.node_fields(t), O.OracleTree(p, f, nf).nodes()
        assert np.array_equal(got["xyz"].view(np.int64), want["xyz"].view(np.int64))
        for k in want:
            assert np.array_equal(got[k], want[k]), k
    finally:
        N.destroy(t)


@pytest.mark.parametrize("kind", ["uniform", "lattice", "plane", "duplicates"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 47, 48, 49, 50, 97, 98, 99, 1023, 1024,
                               1025, 2047, 2048, 2049, 2050, 4099, 12345])
def test_subtree_sizes(n, kind):
    """Base cases, the sequential and the parallel variance, and segments at
    and next to the largest that is finished in shared memory."""
    rs = np.random.RandomState(n)
    p = rs.rand(n, 3)
    if kind == "lattice":  # equal variances and ties along every axis
        p = np.unique(rs.randint(0, 16, (2 * n, 3)), axis=0)[:n] / 16.0
        p = p[rs.permutation(len(p))]
    elif kind == "plane":  # one coordinate constant, one with few values
        p[:, 0], p[:, 1] = -2.5, np.floor(8 * p[:, 1])
    elif kind == "duplicates":
        p = p[rs.randint(0, (n + 1) // 2, n)]
    _check(p, rs.randint(0, 3, len(p)).astype(np.int32), 3)


def _wide(kind, n, rs):
    p = rs.rand(n, 3)
    if kind == "scales":  # twelve decades, both signs: many points on a key
        p = 10.0 ** (-12 * p) * np.where(rs.rand(n, 3) < 0.5, -1, 1)
    elif kind == "outlier":  # all others on one key
        p[n // 3] = [1e300, -1e300, 1e300]
    elif kind == "overflow":
        p[n // 3], p[n // 2] = 1.7e308, -1.7e308
    elif kind == "infinite":
        p[n // 3, 0], p[n // 2, 1], p[n // 5, 2] = np.inf, -np.inf, np.inf
    elif kind == "float32":  # ties along one axis, few and short
        p = p.astype(np.float32).astype(np.float64)
    elif kind == "columns":  # runs of equal x, longer than those put right in place
        p[:, 0] = p[rs.randint(0, n // 60, n), 0]
    elif kind == "pairs":  # runs of equal x, of two and three points, then equal y
        p[:, 0] = p[rs.randint(0, n // 2, n), 0]
        p[:, 1] = np.where(rs.rand(n) < 0.5, p[:, 0], p[:, 1])
    elif kind == "zeros":
        p[rs.rand(n) < 0.01] = 0.0
        p[rs.rand(n, 3) < 0.01] = -0.0
    return p[rs.permutation(n)]


@pytest.mark.parametrize("kind", ["scales", "outlier", "overflow", "infinite", "float32", "columns",
                                  "pairs", "zeros"])
@pytest.mark.parametrize("n", [200, 4096, 4097, 70001])
def test_orders_of_wide_keys(n, kind):
    """The three orders by 32-bit keys, at both sorts and with every rule for a
    key's bits; the general path is the oracle's comparison of all 64."""
    rs = np.random.RandomState(n)
    p = _wide(kind, n, rs)
    f = np.zeros(n, np.int32)
    if kind == "zeros":  # at most 255 copies of a point are a valid tree
        _, first = np.unique(p, axis=0, return_index=True)
        p, f = p[np.sort(first)], f[:len(first)]
    _check(p, f, 1)


@pytest.mark.parametrize("kind", ["uniform", "scales", "outlier", "overflow", "infinite", "columns",
                                  "zeros", "copies", "tight", "line"])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 200, 4096, 4097, 20001])
def test_query_points(n, kind):
    """Points ordered along a curve against the oracle's exhaustive counts (up
    to 4097 points) and against the counts of a tree of the same points."""
    rs = np.random.RandomState(n)
    m = max(n, 60)
    if kind == "copies":  # more than a tree accepts
        q = rs.rand(1 + m // 300, 3)[rs.randint(0, 1 + m // 300, m)][:n]
    elif kind == "tight":  # below the curve's cells
        q = (rs.rand(8, 3)[rs.randint(0, 8, m)] + 1e-9 * rs.rand(m, 3))[:n]
    elif kind == "line":
        q = (rs.rand(m, 1) * [[1.0, 0.0, -2.0]] + [[0.0, 3.0, 0.0]])[:n]
    else:
        q = _wide(kind, m, rs)[:n]
    f = rs.randint(0, 3, n).astype(np.int32)
    scale = {"overflow": 1e308, "outlier": 1.0, "tight": 1e-9}.get(kind, 0.3)
    radii = np.array([0.1, 0.3, 1.0, 4.0]) * scale
    tp = np.concatenate([q[: n // 2 + 1], rs.rand(300, 3)])
    tp = tp[np.unique(tp, axis=0, return_index=True)[1]]
    tf = rs.randint(0, 3, len(tp)).astype(np.int32)
    t = N.build_tree(tp, tf, 3)
    try:
        for mode in (N.KD_MODE_MIXED, N.KD_MODE_FP64):
            got = N.count_points(t, q, f, 3, radii, mode=mode)
            if n <= 4097:
                want = O.OracleTree(tp, tf, 3).brute_counts(q, f, 3, radii, nthreads=4)
                assert np.array_equal(got, want), mode
            elif kind not in ("copies", "zeros"):
                tq = N.build_tree(q, f, 3)
                try:
                    assert np.array_equal(got, N.count_radii(t, tq, radii, mode=mode)), mode
                finally:
                    N.destroy(tq)
    finally:
        N.destroy(t)


@pytest.mark.parametrize("kind", ["uniform", "sky", "scales", "outlier", "infinite", "lattice", "copies",
                                  "uneven"])
@pytest.mark.parametrize("n", [63, 65, 129, 1920, 1921, 2049, 3841, 6000, 9001])
def test_counting_order(n, kind):
    """Trees of one and of several cells, with cells made uneven by copies up
    to the number at which they are no longer the tree's own, against the
    oracle's exhaustive counts: crossed, and symmetric where no point has
    copies of other fields."""
    rs = np.random.RandomState(n)
    if kind == "sky":
        p = rs.randn(n, 3)
        p /= np.sqrt((p * p).sum(1))[:, None]
    elif kind == "lattice":
        p = rs.randint(0, 12, (n, 3)) / 12.0
    elif kind == "copies":  # 250 of each
        p = np.repeat(rs.rand((n + 249) // 250, 3), 250, axis=0)[:n]
    elif kind == "uneven":  # 100 of the points in one corner, as many as fit
        p = rs.rand(n, 3)
        k = min(100, n // 50)
        p[: 40 * k] = np.repeat(0.05 * rs.rand(k, 3), 40, axis=0)
    else:
        p = _wide(kind, n, rs)
    p = p[rs.permutation(n)]
    radii = np.array([0.02, 0.1, 0.3, 0.9])
    fields = np.minimum((np.abs(p[:, 0]) * 3), 2).astype(np.int32)
    mixed = rs.randint(0, 3, n).astype(np.int32)
    for f in (fields, mixed):
        t = N.build_tree(p, f, 3)
        try:
            want = O.OracleTree(p, f, 3).brute_counts(p, f, 3, radii, nthreads=4)
            for mode in (N.KD_MODE_MIXED, N.KD_MODE_FP64):
                assert np.array_equal(N.count_radii(t, t, radii, mode=mode), want), mode
            pq, fq = np.ascontiguousarray(p[::2]), np.ascontiguousarray(f[::2])
            q = N.build_tree(pq, fq, 3)
            try:
                want = O.OracleTree(p, f, 3).brute_counts(pq, fq, 3, radii, nthreads=4)
                assert np.array_equal(N.count_radii(t, q, radii), want)
            finally:
                N.destroy(q)
        finally:
            N.destroy(t)


@pytest.mark.parametrize("n", [174_762, 174_763, 349_525, 349_526, 700_001])
def test_transfer_sizes(n):
    """Inputs and node arrays one short of, at and past the sizes at which
    their copies are staged and cut (4 MB, 8 MB, several pieces)."""
    rs = np.random.RandomState(n)
    p = rs.rand(n, 3)
    _check(p, (p[:, 1] * 5).astype(np.int32), 5)

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

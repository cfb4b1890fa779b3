"""bench.py's CPU baseline where the reference is not built: the oracle stands in
for small workloads of the GPU arm, and for nothing else."""
import pytest

import bench
from oracle import oracle as O


class _Counts:
    """The GPU module's calls that the baseline makes, on the oracle."""
    build_tree = staticmethod(lambda p, f, nf: O.OracleTree(p, f, nf))
    destroy = staticmethod(lambda t: None)

    @staticmethod
    def count_points(t, q, qf, nf, radii):
        return t.brute_counts(q, qf, nf, radii)


class _Wrong(_Counts):
    @staticmethod
    def count_points(t, q, qf, nf, radii):
        return t.brute_counts(q, qf, nf, radii) + 1


@pytest.fixture
def small(monkeypatch):
    monkeypatch.setattr(O, "ref_available", lambda: False)
    return bench.wl_clustered3d(0.002)


def test_oracle_stands_in(small):
    cb = bench.cpu_baseline(small, n_queries=100, gpu=_Counts)
    assert set(cb) >= {"value", "unit", "cores", "kind", "sample", "full_result_s_extrapolated"}
    assert cb["kind"] == "oracle" and "oracle" in cb["note"] and cb["value"] > 0
    assert cb["gpu_counts_equal_reference_on_sample"] is True
    assert bench.cpu_baseline(small, n_queries=100, gpu=_Wrong)["gpu_counts_equal_reference_on_sample"] is False


def test_not_for_the_reference_arm_nor_large_catalogs(small, monkeypatch):
    assert bench.cpu_baseline(small, n_queries=100)["value"] is None
    monkeypatch.setattr(bench, "ORACLE_POINTS", 1000)
    cb = bench.cpu_baseline(small, n_queries=100, gpu=_Counts)
    assert cb["value"] is None and cb["unavailable"]

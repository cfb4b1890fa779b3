"""bench.py's traffic figure follows the workload's own records, not its pairs."""
import types

import bench


class _One:
    local = 0


def _measured(pairs, entries):
    form = dict(pairs=pairs, tile_launches=2, tiles_ms=2.0, dev_ms=2.0, edge_pairs=2 * pairs,
                accepted=0, one_bin_multifield=0, trav_ms=0.1, rechecked=0, launches=6, entries=entries)
    return dict(mixed=form, fp64=form, pairs=pairs, dev_s=2e-3, fpairs=pairs, fdev_s=2e-3, e_wall=1.0,
                e_pairs=pairs, rechecked=0, exact=True, build_s=0.1, h2d=1, d2h=1, pinned=True,
                build_stats={}, e2e_count_s=0.1, clocks={"sm_mhz": 1965.0})


def test_traffic_from_records_and_points():
    w = types.SimpleNamespace(catalogs={"D": ([0] * 1000, None, 1), "R": ([0] * 3000, None, 1)},
                              jobs=[("DR", "R", "D")])
    few, many = (bench._summary(w, _measured(10 ** 9, n), 2, 60.0, 30.0, _One())["roofline"]["traffic"]
                 for n in (2 * 10 ** 5, 2 * 10 ** 6))
    assert few == 16 * 10 ** 5 + 48 * 4000 and many == 16 * 10 ** 6 + 48 * 4000
    # the captured launch: 8.73M records, 1M points, 0.193 GB
    assert abs(16 * 8.73e6 + 48 * 1e6 - 0.193e9) < 0.03 * 0.193e9

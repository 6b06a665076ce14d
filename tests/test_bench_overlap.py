"""CPU test of the bench's factorization rates where the fill ran beside the
randomized re-expansions: no part's time is then that of its work alone."""
import numpy as np

import bench


def test_overlapping_parts_have_no_rate_of_their_own():
    # FIRST 4 x 10, LAST 5 x 3, DENSE 2 x 2
    table = np.array([[0, 4, 10, 0], [2, 5, 3, 40], [3, 2, 2, 55]], np.int64)
    st = {"fillMs": 2.0, "reexpSmemMs": 0.5, "reexpGlobalMs": 0.0, "sketchMs": 6.0,
          "factorMs": 7.0, "reexpSvds": 1, "numSketched": 0}
    w = bench.factorization_work(table, st)
    svd = 22 * 4 ** 3 + 16 * 16 * 10
    assert w["fill_evals_per_s"] is None
    assert np.isclose(w["fill_overlap_ms"], 1.5)
    assert np.isclose(w["kernel_evals_per_s"], (19 + 16 + 40) / 7e-3)
    assert np.isclose(w["reference_equivalent_tflops"], svd / 7e-3 / 1e12)
    # one after the other: the rates of the parts
    w = bench.factorization_work(table, dict(st, factorMs=8.5))
    assert w["fill_evals_per_s"] == 19 / 2e-3 and w["fill_overlap_ms"] == 0.0
    assert np.isclose(w["reference_equivalent_tflops"], svd / 6.5e-3 / 1e12)

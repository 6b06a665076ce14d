"""A right-hand side's result in the FP64 apply does not depend on the other
right-hand sides beside it (bfg_fixed.cu)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402


@pytest.mark.parametrize("R", [2, 7, 16])
@pytest.mark.parametrize("leaf", [64, 4096])
def test_a_right_hand_side_does_not_depend_on_its_neighbours(R, leaf):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 700
    pts = B.curve_points("ellipse", n)
    fac = B.FacHelm2.make_multilevel(B.Helm2(9.0), B.Quadtree(pts, leaf_size=leaf),
                                     B.Quadtree(pts, leaf_size=leaf),
                                     context=B.default_context(0))

    def apply(X):
        return fac.apply(torch.from_numpy(X).cuda()).cpu().numpy()

    X = B.Rng(R + 20).complex_randn(n * R).reshape(n, R)
    y = apply(X)
    u = np.random.RandomState(R).rand(n)
    for other in (complex(np.nan, 0.0), complex(np.inf, 1.0), 2.0 ** -1030, 0.0,
                  2.0 ** np.floor(60 * u), 2.0 ** (90.0 * (np.arange(n) > n // 2))):
        for q in range(R):
            Z = X * (other if np.isscalar(other) else other[:, None])
            Z[:, q] = X[:, q]
            assert np.array_equal(apply(Z)[:, q], y[:, q])

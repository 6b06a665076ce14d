"""Double-float applies of one to five right-hand sides (bfg_df64.cu) on
problems whose stages take 4 and 8 warps an item, and on both sides of the rule
that gives three right-hand sides to the FP64 apply: within 1e-12 of the FP64
apply (a product of ~48 bits, 2^-47, a few hundred of them a row, growth of the
factors included)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402


@pytest.fixture(scope="module", params=[(700, "ellipse", 4096, 1), (1500, "star", 64, 1),
                                        (4096, "ellipse", 64, 1), (2100, "circle", 64, 5)])
def fac(request):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, curve, leaf, problems = request.param
    if problems == 1:
        return B.FacHelm2.make_multilevel(
            B.Helm2(n / 128.0), B.Quadtree(B.uniform_square_points(n, 5), leaf_size=leaf),
            B.Quadtree(B.curve_points(curve, n), leaf_size=leaf), rank_eps=1e-10, pinv_tol=1e-10,
            context=B.default_context(0))
    sizes = [n - 37 * j for j in range(problems)]
    return B.make_batched(B.Helm2(1.0), [(B.uniform_square_points(m, m), B.curve_points(curve, m))
                                         for m in sizes], [m / 30.0 for m in sizes],
                          leaf_size=leaf, rank_eps=1e-10, pinv_tol=1e-10)


@pytest.mark.parametrize("R", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("original", [False, True])
def test_double_float_is_within_its_bound(fac, R, original):
    n = fac.shape[1]
    X = torch.from_numpy(B.Rng(R).complex_randn(n * R).reshape(n, R)).cuda()
    y = fac.apply(X, precision="df64", original_order=original)
    z = fac.apply(X, original_order=original)
    assert torch.linalg.norm(y - z) <= 1e-12 * torch.linalg.norm(z)
    # a right-hand side of its own: the same factors, in another order of sums
    for q in range(R):
        one = fac.apply(X[:, q].contiguous(), precision="df64", original_order=original)
        assert torch.linalg.norm(y[:, q] - one) <= 1e-12 * torch.linalg.norm(one)

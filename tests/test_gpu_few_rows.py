"""Few rows with very many right-hand sides, whose input copy and last sum
split the right-hand sides between thread blocks (bfg_kernels.cu): the same
bits as the columns in groups that do not."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402


@pytest.mark.parametrize("n", [5, 40, 203])
@pytest.mark.parametrize("prec", ["fp64", "fp32", "bf16x3"])
def test_columns_do_not_depend_on_their_number(n, prec):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    fac = B.FacHelm2.make_multilevel(
        B.Helm2(2.0), B.Quadtree(B.uniform_square_points(n, n), leaf_size=16),
        B.Quadtree(B.curve_points("circle", n), leaf_size=16), context=B.default_context(0))
    R, G = 4133, 704   # groups of whole tiles of 8, 16 and 32 columns, both sides with as many
    # outputs as no warps share a row's terms for
    X = torch.from_numpy(B.Rng(n).complex_randn(n * R).reshape(n, R)).cuda()
    if prec != "fp64":
        X = X.to(torch.complex64)
    for original in (False, True):
        y = fac.apply(X, precision=prec, original_order=original)
        for r in range(0, R - G, G):
            part = fac.apply(X[:, r:r + G].contiguous(), precision=prec, original_order=original)
            assert torch.equal(y[:, r:r + G], part)

"""The FP64 apply on operands whose entries differ widely, against the sum of
moduli of each result's own products (bfg_fixed.cuh: fixEven).

Bounds.  Plain FP64: a part of a result is a sum of 2 n products with one
rounding each and a few sums of partial sums, less than (2 n + 16) 2^-53 of the
sum of moduli a part, (2 n + 16) 2^-52 for both.  Fixed point: N 2^-43 of it for
a block of N columns, whatever the entries; where one of the operands' columns
or fewer than an eighth of them are large, or the gradings are opposite and 2^24
or more, the plain form is taken."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402
from test_gpu_fixed import LD, _apply, _dense_blocks  # noqa: E402


def _sums(fac, blocks, X):
    Y = np.zeros((fac.shape[0], X.shape[1]), LD)
    S = np.zeros(Y.shape, np.longdouble)
    for r, c, A in blocks:
        m, n = A.shape
        x = X[c:c + n].astype(LD)
        Y[r:r + m] += A.astype(LD) @ x
        S[r:r + m] += np.abs(A).astype(np.longdouble) @ np.abs(x)
    return Y, S


def _fac(helm, src, tgt, nrm=None):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    fac = B.FacHelm2.make_multilevel(helm, B.Quadtree(src, nrm, leaf_size=4096),
                                     B.Quadtree(tgt, leaf_size=4096),
                                     context=B.default_context(0))
    return fac, _dense_blocks(fac)


@pytest.fixture(scope="module")
def onto_itself():
    """A curve onto itself: the kernel is 0 at r = 0, so the row of a source
    has a structural zero where that source's entry is multiplied."""
    pts = B.curve_points("ellipse", 300)
    return _fac(B.Helm2(9.0), pts, pts)


@pytest.mark.parametrize("R", [1, 2, 16])
@pytest.mark.parametrize("power", [30, 60])
def test_small_entries_beside_a_large_one_that_meets_a_zero(onto_itself, R, power):
    fac, blocks = onto_itself
    n = fac.shape[1]
    X = B.Rng(R).complex_randn(n * R).reshape(n, R)
    for q in range(R):
        X[(37 * q + 11) % n, q] *= 2.0 ** power
    Y, S = _sums(fac, blocks, X)
    err = np.abs(_apply(fac, X).astype(LD) - Y)
    assert np.all(err <= (2 * n + 16) * 2.0 ** -52 * S)


@pytest.mark.parametrize("R", [1, 2, 16])
@pytest.mark.parametrize("spread", ["even", "half", "tenth"])
def test_inputs_of_many_magnitudes(onto_itself, R, spread):
    fac, blocks = onto_itself
    n = fac.shape[1]
    X = B.Rng(R + 7).complex_randn(n * R).reshape(n, R)
    u = np.random.RandomState(R).rand(n, R)
    p = {"even": 60.0 * u, "half": 50.0 * (u < 0.5), "tenth": 50.0 * (u < 0.1)}[spread]
    X *= 2.0 ** np.floor(p)
    Y, S = _sums(fac, blocks, X)
    err = np.abs(_apply(fac, X).astype(LD) - Y)
    assert np.all(err <= n * 2.0 ** -43 * S)


@pytest.mark.parametrize("R", [1, 2, 4, 5, 16])
@pytest.mark.parametrize("n", [5, 31, 130, 500])
def test_operands_graded_in_opposite_directions(n, R):
    """A double layer on a line whose normals turn away from it by 2^-g t: a
    column's entries have that factor.  Inputs with the opposite one, so that
    every product is of like size; every block has the whole range."""
    t = np.random.RandomState(n).permutation(n) / max(1, n - 1.0)
    src = np.stack([np.linspace(0.0, 1.0, n), np.zeros(n)], 1)
    tgt = np.stack([np.linspace(1.5, 2.5, 70), np.zeros(70)], 1)
    X0 = B.Rng(n).complex_randn(n * R).reshape(n, R)
    for g in (6.0, 12.0, 24.0, 40.0, 60.0):
        nrm = np.stack([2.0 ** (-g * t), np.ones(n)], 1)
        fac, blocks = _fac(B.Helm2(9.0, B.LayerPot.PvDouble), src, tgt, nrm)
        X = X0 * (2.0 ** (g * t))[fac.src_perm, None]
        Y, S = _sums(fac, blocks, X)
        err = np.abs(_apply(fac, X).astype(LD) - Y)
        bound = (2 * n + 16) * 2.0 ** -52 if g >= 24.0 and n > 100 else n * 2.0 ** -43
        assert np.all(err <= bound * S), (g, float((err / S).max()))

"""The FP64 apply's fixed-point products (bfg_fixed.cu) against extended
precision, evaluated from the factorization's own stored blocks.

Every block is dense here (no split below depth 1), so a row's error bound is
known: a part of an entry is off by at most 2^-55 of its row's largest part
(2^-54 of the largest input, whose scale may start a binade high), a complex
product has two such real products a part, and each FP64 rounding of a sum is
below 2^-53 of the sum of moduli.  Together less than
2^-51 n max|a_i| max|x| a block of n columns."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402

LD = np.clongdouble


def _dense_blocks(fac):
    """(row offset, column offset, block) of every block of an all-dense plan."""
    tab, ent = fac.blocks()
    lines = [ln.split() for ln in fac.describe().splitlines()]
    assert lines[0][0] == "BD" and all(ln[0] == "DC" for ln in lines[3:])
    ro, co = [int(v) for v in lines[1][1:]], [int(v) for v in lines[2][1:]]
    out, nc = [], len(co) - 1
    for b, (kind, m, n, off) in enumerate(tab):
        assert kind == 3
        out.append((ro[b // nc], co[b % nc], ent[off:off + m * n].reshape(n, m).T))
    return out


def _problem(m, n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    fac = B.FacHelm2.make_multilevel(
        B.Helm2(9.0), B.Quadtree(B.uniform_square_points(n, m), leaf_size=4096),
        B.Quadtree(B.curve_points("circle", m), leaf_size=4096), context=B.default_context(0))
    return fac, _dense_blocks(fac)


def _exact_and_bound(fac, blocks, X):
    Y = np.zeros((fac.shape[0], X.shape[1]), LD)
    bound = np.zeros(Y.shape, np.longdouble)
    for r, c, A in blocks:
        m, n = A.shape
        x = X[c:c + n].astype(LD)
        Y[r:r + m] += A.astype(LD) @ x
        bound[r:r + m] += (2.0 ** -51 * n * np.abs(A).max(1).astype(np.longdouble)[:, None]
                           * np.abs(x).max(0)[None, :])
    return Y, bound


def _apply(fac, X):
    return fac.apply(torch.from_numpy(X).cuda()).cpu().numpy()


# quarters of the points land in a block, so these put block rows and columns
# on both sides of the 16-row tiles, the 32-row items, and the 8-, 32-, 64-,
# 120- and 128-column steps, chunks and passes
@pytest.mark.parametrize("m,n", [(4, 4), (9, 31), (66, 33), (131, 127), (130, 257), (70, 485),
                                 (257, 515), (40, 2101)])
def test_fixed_point_error_is_within_its_bound(m, n):
    fac, blocks = _problem(m, n)
    X = B.Rng(n).complex_randn(n * 33).reshape(n, 33)
    X *= np.exp(B.Rng(m).complex_randn(n).real * 3.0)[:, None]   # rows of unlike size
    Y, bound = _exact_and_bound(fac, blocks, X)
    for R in (1, 2, 4, 5, 8, 9, 16, 17, 33):
        y = _apply(fac, X[:, :R].copy())
        err = np.abs(y.astype(LD) - Y[:, :R])
        assert np.all(err <= bound[:, :R]), (R, float((err / bound[:, :R]).max()))


def test_scales_are_exact_and_ranges_fall_back():
    fac, blocks = _problem(90, 300)
    X = B.Rng(1).complex_randn(300 * 9).reshape(300, 9)
    for R in (1, 3, 9):
        y = _apply(fac, X[:, :R].copy())
        for s in (-600.0, 600.0):     # a power of two changes exponents only
            assert np.array_equal(_apply(fac, X[:, :R] * 2.0 ** s), y * 2.0 ** s)
        # right-hand sides of unlike size side by side keep their own scale
        w = 2.0 ** (40.0 * (np.arange(R) - R // 2))
        assert np.array_equal(_apply(fac, X[:, :R] * w), y * w)
        assert not np.any(_apply(fac, np.zeros((300, R), complex)))
        # below the fixed-point range: plain FP64 sums
        Y, bound = _exact_and_bound(fac, blocks, X[:, :R])
        tiny = _apply(fac, X[:, :R] * 2.0 ** -1010) * 2.0 ** 1000 * 2.0 ** 10
        assert np.all(np.abs(tiny.astype(LD) - Y) <= bound + np.abs(Y).max() * 2.0 ** -40)


@pytest.mark.parametrize("R", [1, 2, 7, 16])
def test_infinities_and_nans_reach_the_rows_they_meet(R):
    fac, blocks = _problem(90, 300)
    X = B.Rng(2).complex_randn(300 * R).reshape(300, R)
    clean = _apply(fac, X.copy())
    Y, bound = _exact_and_bound(fac, blocks, X)
    for bad in (complex(np.inf, 0.0), complex(0.0, -np.inf), complex(np.nan, 1.0)):
        Z = X.copy()
        Z[17, R // 2] = bad
        y = _apply(fac, Z)
        assert not np.any(np.isfinite(y[:, R // 2]))
        others = np.arange(R) != R // 2
        assert np.all(np.abs(y[:, others].astype(LD) - Y[:, others]) <= bound[:, others])
    assert np.array_equal(_apply(fac, X.copy()), clean)


# ranks (and so the products' sizes) below, at and above the 32-column and
# 64-row tiles and the 64-row flush interval of the factorization's products
@pytest.mark.parametrize("k", [12.0, 25.0, 41.0, 60.0, 97.0])
def test_factorization_products_match_the_full_path(k):
    """The operators of the randomized path, whose products the digits form,
    and of the full path, which uses none (the bound of the sketch tests)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 2500
    src, tgt = B.uniform_square_points(n, 11), B.curve_points("star", n)
    X = torch.from_numpy(B.Rng(3).complex_randn(2 * n).reshape(n, 2)).cuda()
    y = [B.FacHelm2.make_multilevel(B.Helm2(k), B.Quadtree(src, leaf_size=32),
                                    B.Quadtree(tgt, leaf_size=32), rank_eps=1e-10, pinv_tol=1e-10,
                                    sketch=s, context=B.default_context(0)).apply(X)
         for s in (True, False)]
    assert torch.linalg.norm(y[0] - y[1]) < 2e-9 * torch.linalg.norm(y[1])


def test_small_rank_blocks_solve_the_reexpansion_least_squares():
    """Ranks 8 to 31, which the QR-preconditioned Jacobi at full width takes
    too, against the oracle's pseudo-inverse (the bounds of the sketch tests)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import rel_err
    from oracle import bf_oracle as O
    n, k, tol = 2048, 24.0, 1e-7
    src, tgt = B.uniform_square_points(n, 4), B.curve_points("ellipse", n)
    fac = B.FacHelm2.make_multilevel(B.Helm2(k), B.Quadtree(src, leaf_size=64),
                                     B.Quadtree(tgt, leaf_size=64), rank_eps=tol, pinv_tol=tol,
                                     context=B.default_context(0))
    of = O.Factorization(O.Helm2(k), src, tgt, leaf_size=64, eps=tol, rcut="relative", fill=False)
    tab, ent = fac.blocks()
    ranks = set()
    for (kind, m, nb, off), ob in zip(tab, of.blocks()):
        if kind not in (0, 1) or not 8 <= m < 32 or (m in ranks and len(ranks) < 12):
            continue
        Z = ent[off:off + m * nb].reshape(nb, m).T
        eq, chk = O.circle_points(ob.ceq, m)[0], O.circle_points(ob.cchk, m)[0]
        orig = (of.src_tree_pts[ob.src_range[0]:ob.src_range[1]] if ob.kind == "first"
                else O.circle_points(ob.corig, nb)[0])
        Ze, Zo = (O.kernel_matrix(O.Helm2(k), p, chk) for p in (eq, orig))
        Xo = O.lstsq_pinv(Ze, Zo, "relative", tol)
        assert (np.linalg.norm(Ze @ Z - Zo) < 2 * np.linalg.norm(Ze @ Xo - Zo)
                + 1e-12 * np.linalg.norm(Zo))
        assert rel_err(Z, Xo) < 1e-6
        ranks.add(m)
    assert len(ranks) >= 6


@pytest.mark.parametrize("m,n", [(9, 31), (131, 127), (130, 257), (70, 515)])
def test_fp32_tiles_are_within_their_bound(m, n):
    """The FP32 apply of several right-hand sides (bfg_kernels.cu): every
    tile width and its remainders, against extended precision.  FP32 entries
    and inputs are off by 2^-24 of themselves and every product and sum rounds
    to FP32: less than 2^-22 sum |a||x| (n + 8) / 4 a block of n columns."""
    fac, blocks = _problem(m, n)
    X = B.Rng(n).complex_randn(n * 33).reshape(n, 33).astype(np.complex64)
    Y = np.zeros((m, 33), LD)
    bound = np.zeros((m, 33))
    for r, c, A in blocks:
        x = X[c:c + A.shape[1]]
        Y[r:r + A.shape[0]] += A.astype(LD) @ x.astype(LD)
        bound[r:r + A.shape[0]] += 2.0 ** -22 * (A.shape[1] + 8) / 4 * (np.abs(A) @ np.abs(x))
    for R in (2, 3, 4, 5, 8, 9, 16, 17, 33):
        y = fac.apply(torch.from_numpy(X[:, :R].copy()).cuda(), precision="fp32").cpu().numpy()
        assert np.all(np.abs(y.astype(LD) - Y[:, :R]) <= bound[:, :R])


@pytest.mark.parametrize("n,onto_itself", [(33, False), (1153, False), (1153, True)])
def test_wide_and_narrow_applies_agree(n, onto_itself):
    """The input copy and the final sum (bfg_kernels.cu) share a row's terms
    between warps or not by the number of outputs and of terms (many for a
    curve onto itself), with every width of their thread blocks: both against the FP64 apply of single columns, whose
    results FP64 repeats to a few units of 2^-51 of the sums of moduli (1e-12
    of the norm with the multi-level factors' growth) and FP32 and three bf16
    planes to a few 1e-6."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from conftest import rel_err
    tgt = B.curve_points("ellipse", n)
    fac = B.FacHelm2.make_multilevel(
        B.Helm2(9.0),
        B.Quadtree(tgt if onto_itself else B.uniform_square_points(n, 3), leaf_size=32),
        B.Quadtree(tgt, leaf_size=32), context=B.default_context(0))
    X = torch.from_numpy(B.Rng(n).complex_randn(n * 130).reshape(n, 130)).cuda()
    for orig in (False, True):
        cols = [fac.apply(X[:, i].contiguous(), original_order=orig).cpu().numpy()
                for i in range(130)]
        exact = np.stack(cols, 1)
        for R in (1, 2, 3, 7, 16, 33, 64, 113, 114, 130):
            for prec, tol in (("fp64", 1e-11), ("fp32", 2e-5), ("bf16x3", 2e-5)):
                x = X[:, :R].to(torch.complex128 if prec == "fp64" else torch.complex64)
                y = fac.apply(x.contiguous(), precision=prec, original_order=orig)
                assert rel_err(y.cpu().numpy().astype(complex), exact[:, :R]) < tol


@pytest.mark.parametrize("n", [485, 1001, 2101, 4321])
def test_plain_sums_of_shared_items(n):
    """One right-hand side whose items' passes clusters of 2 and 4 CTAs share
    (from 2 and 4 passes of 120 columns a block): plain FP64 sums in every
    CTA's passes, and an infinity in the first, a middle and the last column.
    Bounds as above."""
    fac, blocks = _problem(40, n)
    X = B.Rng(n).complex_randn(n).reshape(n, 1)
    Y, bound = _exact_and_bound(fac, blocks, X)
    clean = _apply(fac, X)
    assert np.all(np.abs(clean.astype(LD) - Y) <= bound)
    tiny = _apply(fac, X * 2.0 ** -1010) * 2.0 ** 1000 * 2.0 ** 10
    assert np.all(np.abs(tiny.astype(LD) - Y) <= bound + np.abs(Y).max() * 2.0 ** -40)
    for at in (0, n // 2, n - 1):
        Z = X.copy()
        Z[at] = complex(0.0, np.inf)
        assert not np.any(np.isfinite(_apply(fac, Z)))
    assert np.array_equal(_apply(fac, X), clean)

"""The randomized re-expansion's blocks of several hundred columns at the tight
tolerance (bfg_sketch.cu): their FP32-started Jacobi keeps its rotations' product
in global memory (more than 118 columns) or shared memory, and a product that
were not unitary to FP64 would show as a residual of its size."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import bf_oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402


@pytest.mark.parametrize("n,k,width", [(16384, 500.0, 150), (32768, 2000.0, 500)])
def test_wide_blocks_solve_the_reexpansion_least_squares(n, k, width):
    """Residuals within 2x (+1e-12) of the oracle's pseudo-inverse, the blocks
    within 1e-4 of it (an entry at the cut of 1e-10 moves by 1e-16 / 1e-10
    times a few hundred roundings), the bars of the other re-expansion tests."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    tol = 1e-10
    src, tgt = O.uniform_square_points(n, 7), O.curve_points("ellipse", n)
    fac = B.FacHelm2.make_multilevel(B.Helm2(k), B.Quadtree(src, leaf_size=64),
                                     B.Quadtree(tgt, leaf_size=64), rank_eps=tol, pinv_tol=tol,
                                     context=B.default_context(0))
    st = fac.stats()
    assert st["jacobiNotConverged"] == 0 and st["sketchMaxWidth"] >= width
    of = O.Factorization(O.Helm2(k), src, tgt, leaf_size=64, eps=tol, rcut="relative", fill=False)
    tab, ent = fac.blocks()
    found = sorted([(int(m), i) for i, (kind, m, nb, off) in enumerate(tab) if kind in (0, 1)],
                   reverse=True)
    blocks = of.blocks()
    pick = [next(f for f in found if f[0] <= most) for most in (600, 500, 350, 250, 160, 118)
            if found[-1][0] <= most]
    assert pick[0][0] >= 450
    h = O.Helm2(k)
    for m, i in dict(pick).items():
        _, _, nb, off = tab[i]
        ob = blocks[i]
        Z = ent[off:off + m * nb].reshape(nb, m).T
        eq, chk = O.circle_points(ob.ceq, m)[0], O.circle_points(ob.cchk, m)[0]
        orig = (of.src_tree_pts[ob.src_range[0]:ob.src_range[1]] if ob.kind == "first"
                else O.circle_points(ob.corig, nb)[0])
        Ze, Zo = (O.kernel_matrix(h, p, chk) for p in (eq, orig))
        Xo = O.lstsq_pinv(Ze, Zo, "relative", tol)
        norm = np.linalg.norm(Zo)
        assert np.linalg.norm(Ze @ Z - Zo) < 2 * np.linalg.norm(Ze @ Xo - Zo) + 1e-12 * norm, m
        assert rel_err(Z, Xo) < 1e-4, m

"""The per-iteration kernels of the preconditioners (bfg_solver.cu,
bfg_coarse.cu) on curves of 1 to 131 points: both sides of the 4-row warps and
16-row thread blocks of the block-Jacobi product, of the 8-mode and 32-point
tiles of the coarse restriction and prolongation."""
import ctypes

import numpy as np
import pytest

from conftest import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402

SIZES = [1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 63, 65, 97, 131]


@pytest.fixture(scope="module")
def problem():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    k, r = 12.0, 0.3
    pts, nrm, w, off = [], [], [], [0]
    for i, n in enumerate(SIZES):
        t = 2 * np.pi * np.arange(n) / n
        u = np.stack([np.cos(t), np.sin(t)], 1)
        pts.append(np.array([i % 4, i // 4]) + r * u)
        nrm.append(u)
        w.append(np.full(n, 2 * np.pi * r / n))
        off.append(off[-1] + n)
    pts, nrm, w = np.concatenate(pts), np.concatenate(nrm), np.concatenate(w)
    helm = B.Helm2(k, B.LayerPot.CombinedField, alpha=-1j * k, beta=1.0)
    fac = B.FacHelm2.make_multilevel(helm, B.Quadtree(pts, nrm, leaf_size=64),
                                     B.Quadtree(pts, leaf_size=64), rank_eps=1e-10,
                                     pinv_tol=1e-10, context=B.default_context(0))
    s = B.System(fac, pts, nrm, w, off, kr_order=0, diag_shift=0.5)
    s.build_block_jacobi()
    return s, off, w, k


def test_coarse_correction_of_every_curve_size(problem):
    """Against the same product from the device's A_c^-1 and the Fourier modes
    in FP64: FP32 table, inverse and sums, each rounding 2^-24 of the sums of
    moduli, D + 8 of them at most."""
    s, off, w, k = problem
    D = s.build_coarse(5)
    ainv = s.coarse_matrices()[1].cpu().numpy().astype(complex)
    phi = np.zeros((off[-1], D), complex)
    c = 0
    for o, e in zip(off[:-1], off[1:]):
        q = min(int(np.ceil(k * w[o:e].sum() / (2 * np.pi))) + 5, (e - o - 1) // 2)
        m = np.arange(-q, q + 1)
        phi[o:e, c:c + 2 * q + 1] = np.exp(2j * np.pi * np.outer(np.arange(e - o), m) / (e - o)
                                           ) / np.sqrt(e - o)
        c += 2 * q + 1
    assert c == D
    r = B.Rng(3).complex_randn(off[-1])
    z = s.apply_coarse(torch.from_numpy(r).cuda()).cpu().numpy()
    bound = 2.0 ** -23 * (D + 8) * (np.abs(phi) @ (np.abs(ainv) @ (np.abs(phi).T @ np.abs(r))))
    assert np.all(np.abs(z - phi @ (ainv @ (phi.conj().T @ r))) <= bound)


def test_fp32_block_jacobi_of_every_curve_size(problem):
    """The solve with the FP32 inverses takes the iterations of one with the
    FP64 inverses, to one, and gives the same solution: a wrong row would be a
    wrong preconditioner."""
    s, off, _, _ = problem
    b = torch.from_numpy(B.Rng(4).complex_randn(off[-1])).cuda()

    def fp64_inverses(r, z, stream):
        assert B._solver_sigs().bfgSystemApplyBlockJacobi(s.handle, ctypes.c_void_p(r),
                                                          ctypes.c_void_p(z)) == 0

    x, info = B.solve_gmres(s, b, tol=1e-10, max_num_iter=100, precond="block_jacobi")
    x64, info64 = B.solve_gmres(s, b, tol=1e-10, max_num_iter=100, precond=fp64_inverses)
    assert info["converged"] and abs(info["iterations"] - info64["iterations"]) <= 1
    assert rel_err(x.cpu().numpy(), x64.cpu().numpy()) < 1e-8


@pytest.mark.parametrize("n", [15, 16, 17, 1023, 1024, 1025, 2081])
def test_arnoldi_residual_is_the_true_one(n):
    """One to three row chunks of the Gram-Schmidt kernels and remainders of
    their 16 rows: wrong coefficients or norms would part the residual of the
    Arnoldi relation from that of the solution (both FP64, a few hundred
    roundings of 2^-53 and products within 1e-12)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    k, t = 9.0, 2 * np.pi * np.arange(n) / n
    pts = np.stack([np.cos(t), np.sin(t)], 1)
    helm = B.Helm2(k, B.LayerPot.CombinedField, alpha=-1j * k, beta=1.0)
    fac = B.FacHelm2.make_multilevel(helm, B.Quadtree(pts, pts, leaf_size=64),
                                     B.Quadtree(pts, leaf_size=64), rank_eps=1e-13,
                                     pinv_tol=1e-13, context=B.default_context(0))
    s = B.System(fac, pts, pts, np.full(n, 2 * np.pi / n), [0, n], kr_order=6, diag_shift=0.5)
    b = torch.from_numpy(B.Rng(n).complex_randn(n)).cuda()
    for iters in (3, n):
        x, info = B.solve_gmres(s, b, tol=1e-9, max_num_iter=iters, precond="none")
        res = torch.linalg.norm(b - s.apply(x)).item() / torch.linalg.norm(b).item()
        assert abs(info["trueRelResidual"] - res) < 1e-10
        assert abs(info["relResidual"] - res) < 1e-10
        assert iters == 3 or info["converged"]

"""The preconditioners' kernels on one large curve among many small ones: every
curve's rows and modes are reached, whatever the largest one's size."""
import numpy as np
import pytest

from conftest import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402


@pytest.fixture(scope="module")
def problem():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    k = 6.0
    sizes = [1 + i % 9 for i in range(200)] + [611] + [1 + i % 5 for i in range(150)]
    pts, nrm, w, off = [], [], [], [0]
    for i, n in enumerate(sizes):
        r = 2.0 if n > 100 else 0.05
        centre = (0.0, 0.0) if n > 100 else (3.0 + 0.3 * (i % 19), -3.0 + 0.3 * (i // 19))
        t = 2 * np.pi * np.arange(n) / n
        u = np.stack([np.cos(t), np.sin(t)], 1)
        pts.append(np.array(centre) + r * u)
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


def test_coarse_correction(problem):
    """Against the same product from the device's A_c^-1 and the Fourier modes
    in FP64: FP32 table, inverse and sums, each rounding 2^-24 of the sums of
    moduli, D + 8 of them at most."""
    s, off, w, k = problem
    D = s.build_coarse(3)
    ainv = s.coarse_matrices()[1].cpu().numpy().astype(complex)
    phi = np.zeros((off[-1], D), complex)
    c = 0
    for o, e in zip(off[:-1], off[1:]):
        q = min(int(np.ceil(k * w[o:e].sum() / (2 * np.pi))) + 3, (e - o - 1) // 2)
        m = np.arange(-q, q + 1)
        phi[o:e, c:c + 2 * q + 1] = np.exp(2j * np.pi * np.outer(np.arange(e - o), m) / (e - o)
                                           ) / np.sqrt(e - o)
        c += 2 * q + 1
    assert c == D
    r = B.Rng(3).complex_randn(off[-1])
    z = s.apply_coarse(torch.from_numpy(r).cuda()).cpu().numpy()
    bound = 2.0 ** -23 * (D + 8) * (np.abs(phi) @ (np.abs(ainv) @ (np.abs(phi).T @ np.abs(r))))
    assert np.all(np.abs(z - phi @ (ainv @ (phi.conj().T @ r))) <= bound)


def test_fp32_block_jacobi_of_every_curve(problem):
    """After one iteration the solution is a multiple of M b: curve by curve
    against the FP64 inverses, to 1e-3 (FP32 inverses of well-conditioned
    blocks; a row left out or of another curve is off by its own size)."""
    s, off, _, _ = problem
    b = torch.from_numpy(B.Rng(4).complex_randn(off[-1])).cuda()
    x, _ = B.solve_gmres(s, b, tol=1e-12, max_num_iter=1, precond="block_jacobi")
    z = torch.empty_like(b)
    torch.cuda.synchronize()
    assert B._solver_sigs().bfgSystemApplyBlockJacobi(s.handle, B._VP(b.data_ptr()),
                                                      B._VP(z.data_ptr())) == 0
    torch.cuda.synchronize()
    x, z = x.cpu().numpy(), z.cpu().numpy()
    x *= np.vdot(x, z) / np.vdot(x, x)
    for o, e in zip(off[:-1], off[1:]):
        assert rel_err(x[o:e], z[o:e]) < 1e-3


def test_solutions_agree(problem):
    s, off, _, _ = problem
    s.build_coarse(3)
    b = torch.from_numpy(B.Rng(4).complex_randn(off[-1])).cuda()
    x, info = B.solve_gmres(s, b, tol=1e-10, max_num_iter=120, precond="two_level")
    z, plain = B.solve_gmres(s, b, tol=1e-10, max_num_iter=1000, precond="none")
    assert info["converged"] and plain["converged"]
    assert info["iterations"] < plain["iterations"]
    assert rel_err(x.cpu().numpy(), z.cpu().numpy()) < 1e-6

"""The work that users of butterfly_gb300 have it do, as measurable cases.

Three kinds of call make up the framework's use:

* ``make``   factorize the Helmholtz kernel between two point sets (one problem
             or a batch of uneven ones) and apply the result to its first
             right-hand sides;
* ``apply``  multiply right-hand sides by a factorization that the program
             keeps: device tensors or host arrays, one vector to hundreds,
             every precision, tree order or the points' own order;
* ``solve``  FGMRES on a combined-field scattering operator whose
             factorization, preconditioner and right-hand side are at hand.

Geometries, wavenumbers (about n / 128 for n points, so that the points per
wavelength stay the same), leaf size and tolerances are those of the
repository's benchmark and tests.
"""
import functools
import math

import numpy as np
import torch

import butterfly_gb300 as B

LEAF = 64
KR6 = (4.967362978287758, -16.20501504859126, 25.85153761832639,
       -22.22599466791883, 9.930104998037539, -1.817995878141594)
C128 = ("fp64", "df64")
ENTRY_BYTES = {"fp64": 16, "df64": 16, "fp32": 8, "bf16x2": 8, "bf16x3": 12}


def _make(name, n, k, curve, tol, problems=1, rhs=1, precision="fp64"):
    return dict(name=name, kind="make", n=n, k=k, curve=curve, tol=tol, problems=problems,
                rhs=rhs, precision=precision)


def _apply(name, n, k, curve, tol, rhs, precision, problems=1, original=False, host=False):
    return dict(name=name, kind="apply", n=n, k=k, curve=curve, tol=tol, problems=problems,
                rhs=rhs, precision=precision, original=original, host=host)


def _solve(name, circles, k, precond, precision):
    return dict(name=name, kind="solve", circles=circles, k=k, precond=precond,
                precision=precision)


def listed():
    return [
        # a first factorization and product of a small problem: the smallest
        # benchmark configuration, what a user tries first
        _make("make_small", 4096, 64.0, "circle", 1e-8),
        # a production factorization at the tight tolerance, and its first product
        _make("make_large", 65536, 512.0, "ellipse", 1e-10),
        # many independent problems of uneven size factorized at once (n is
        # the largest; sizes log-uniform from 1,024), 8 right-hand sides each
        _make("make_batched", 16384, 0.0, "circle", 1e-8, problems=12, rhs=8),
        # one small matrix-vector product in the default precision: a Krylov
        # method's inner call, where launches count
        _apply("matvec_small", 4096, 64.0, "circle", 1e-8, 1, "fp64"),
        # the same at production size
        _apply("matvec_large", 65536, 512.0, "ellipse", 1e-10, 1, "fp64", original=True),
        # a block of right-hand sides in the reference's arithmetic
        _apply("apply_fp64_16", 65536, 512.0, "ellipse", 1e-10, 16, "fp64"),
        # a batch of problems, 8 right-hand sides, single precision
        _apply("batched_fp32_8", 16384, 0.0, "circle", 1e-8, 8, "fp32", problems=12),
        # a few right-hand sides on a ragged mid-size problem, in the points' order
        _apply("apply_bf16x3_5", 10007, 80.0, "star", 1e-7, 5, "bf16x3", original=True),
        # many right-hand sides at 1e-6: the throughput workload
        _apply("apply_bf16x3_256", 65536, 512.0, "star", 1e-7, 256, "bf16x3"),
        # host arrays in and out: the drop-in for the reference's bfMatMul
        _apply("apply_host_16", 32768, 256.0, "ellipse", 1e-10, 16, "fp64", host=True),
        # a scattering solve with the reference's preconditioner
        _solve("gmres_block_jacobi", 16, 100.0, "block_jacobi", "fp64"),
        # the larger scattering solve with the two-level preconditioner and
        # double-float products
        _solve("gmres_two_level", 64, 200.0, "two_level", "df64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["make", "apply", "apply", "apply", "apply", "solve"])
    if kind == "solve":
        c = _solve("", rng.randint(8, 40), round(rng.uniform(60.0, 180.0), 3),
                   rng.choice(["block_jacobi", "two_level"]), rng.choice(["fp64", "df64"]))
    else:
        n = _log_int(rng, 1024, 49152)
        k = round(n / 128.0 * rng.uniform(0.7, 1.3), 3)
        curve = rng.choice(["circle", "ellipse", "star"])
        tol = rng.choice([1e-7, 1e-8, 1e-10])
        problems = rng.choice([1, 1, 1, 1, 5, 9])
        if problems > 1:
            n, k = min(n, 12000), 0.0
        if kind == "make":
            c = _make("", n, k, curve, tol, problems, rng.choice([1, 3, 8]))
        else:
            precision = rng.choice(["fp64", "fp64", "bf16x3", "bf16x3", "fp32", "df64", "bf16x2"])
            c = _apply("", n, k, curve, tol, rng.choice([1, _log_int(rng, 2, 16),
                                                         _log_int(rng, 17, 256)]),
                       precision, problems, rng.random() < 0.5, rng.random() < 0.15)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _problems(case, seed):
    """(src, tgt, k) of every problem: sources uniform in [-1, 1]^2, targets
    equispaced on the curve around them.  The sizes belong to the case, the
    points to the seed."""
    P = case["problems"]
    if P == 1:
        sizes, ks = [case["n"]], [case["k"]]
    else:
        u = np.random.RandomState(P).rand(P)
        lo, hi = math.log(min(1024, case["n"])), math.log(case["n"])
        sizes = [int(math.exp(lo + (hi - lo) * v)) for v in u]
        ks = [n / 30.0 for n in sizes]
    # targets: a circle of radius 3, an ellipse (3, 2), a star around radius 3
    return [(B.uniform_square_points(n, 1000 * seed + j), B.curve_points(case["curve"], n), k)
            for j, (n, k) in enumerate(zip(sizes, ks))]


def _factorize(case, problems):
    tol = case["tol"]
    if case["problems"] == 1:
        src, tgt, k = problems[0]
        return B.FacHelm2.make_multilevel(B.Helm2(k), B.Quadtree(src, leaf_size=LEAF),
                                          B.Quadtree(tgt, leaf_size=LEAF), rank_eps=tol,
                                          pinv_tol=tol)
    return B.make_batched(B.Helm2(1.0), [(s, t) for s, t, _ in problems],
                          [k for _, _, k in problems], leaf_size=LEAF, rank_eps=tol,
                          pinv_tol=tol, tree_on_gpu=True)


def _rhs(n, R, precision, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((n, R, 2), generator=g, device="cuda", dtype=torch.float64)
    x = torch.view_as_complex(x)
    if R == 1:
        x = x[:, 0].contiguous()
    return x if precision in C128 else x.to(torch.complex64)


def _scattering(case, seed):
    # the layout belongs to the case (it sets the number of unknowns), the
    # incident wave to the seed
    k = case["k"]
    pts, nrm, w, off, _ = B.scattering_geometry(num=case["circles"], k=k, ppw=12.0, rmin=0.05,
                                                rmax=0.15, box=2.0, gap=0.05, seed=0)
    theta = 2 * np.pi * np.random.RandomState(seed).rand()
    b = -np.exp(1j * k * (pts @ np.array([np.cos(theta), np.sin(theta)])))
    return pts, nrm, w, off, torch.from_numpy(b).cuda()


def prepare(case, seed):
    if case["kind"] == "solve":
        k = case["k"]
        pts, nrm, w, off, b = _scattering(case, seed)
        helm = B.Helm2(k, B.LayerPot.CombinedField, alpha=-1j * k, beta=1.0)
        fac = B.FacHelm2.make_multilevel(helm, B.Quadtree(pts, nrm, leaf_size=LEAF),
                                         B.Quadtree(pts, leaf_size=LEAF), rank_eps=1e-10,
                                         pinv_tol=1e-10)
        system = B.System(fac, pts, nrm, w, off, kr_order=6, diag_shift=0.5)
        system.build_block_jacobi()
        if case["precond"] == "two_level":
            system.build_coarse(5)
        system.set_apply_precision(case["precision"])
        return dict(case=case, system=system, b=b)
    problems = _problems(case, seed)
    n = sum(len(s) for s, _, _ in problems)
    x = _rhs(n, case["rhs"], case["precision"], seed)
    if case["kind"] == "make":
        return dict(case=case, problems=problems, x=x)
    fac = _factorize(case, problems)
    fac.prepare(case["precision"])
    if case["host"]:
        x = x.to(torch.complex128).cpu().numpy()
    return dict(case=case, fac=fac, x=x)


def run(state):
    case = state["case"]
    if case["kind"] == "make":
        fac = _factorize(case, state["problems"])
        return fac.apply(state["x"], precision=case["precision"], original_order=True)
    if case["kind"] == "apply":
        return state["fac"].apply(state["x"], precision=case["precision"],
                                  original_order=case["original"])
    iters = 1000 if case["precond"] == "block_jacobi" else 300
    x, _ = B.solve_gmres(state["system"], state["b"], tol=1e-8, max_num_iter=iters,
                         precond=case["precond"])
    return x


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _plan_entries(k, src, tgt, tol):
    total = 0
    for line in B.plan_helm2(k, src, tgt, LEAF, tol)[2].splitlines():
        f = line.split()
        if f[0] in ("B", "DC"):
            total += int(f[-2]) * int(f[-1])   # rows, columns of a stored block
    return total


@functools.lru_cache(maxsize=64)
def _entries(items):
    """Stored complex entries of the factorization (its block structure)."""
    case = dict(items)
    if case["kind"] == "solve":
        pts = B.scattering_geometry(num=case["circles"], k=case["k"], seed=0)[0]
        return len(pts), _plan_entries(case["k"], pts, pts, 1e-10)
    problems = _problems(case, 0)
    return (sum(len(s) for s, _, _ in problems),
            sum(_plan_entries(k, s, t, case["tol"]) for s, t, k in problems))


def work(case):
    n, entries = _entries(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    if case["kind"] == "solve":
        # products with the operator that the solves of these sizes take
        # (iterations, the starting and the final residual)
        products = 8 if case["precond"] == "two_level" else 50
        return dict(bytes=products * (16.0 * entries + 48.0 * n), flops=products * 8.0 * entries)
    R, elem = case["rhs"], 16 if case["precision"] in C128 else 8
    if case["kind"] == "make":
        # points in, every stored entry written and read once; at least one
        # kernel value (two Bessel functions, about 100 operations) an entry
        return dict(bytes=64.0 * n + 32.0 * entries + 2.0 * elem * n * R,
                    flops=(100.0 + 8.0 * R) * entries)
    if case["host"]:
        elem = 16
    return dict(bytes=float(ENTRY_BYTES[case["precision"]]) * entries + 2.0 * elem * n * R,
                flops=8.0 * R * entries)


# ---------------------------------------------------------------------------
# the same products and solutions from the dense kernel in 64 bits
# ---------------------------------------------------------------------------
def _tree_orders(case, problems):
    """Concatenated source and target permutations of the problems' trees."""
    sp, tp, base = [], [], 0
    for src, tgt, k in problems:
        p = B.quadtree_build([src, tgt], leaf_size=LEAF)
        sp.append(p[0][0] + base)
        tp.append(p[1][0] + base)
        base += len(src)
    return (torch.from_numpy(np.concatenate(sp)).cuda(), torch.from_numpy(np.concatenate(tp)).cuda())


def _dense_apply(src, tgt, k, x, rows=2048):
    s, t = torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda()
    out = torch.empty((len(tgt), x.shape[1]), dtype=torch.complex128, device="cuda")
    for i in range(0, len(tgt), rows):
        r = k * torch.hypot(t[i:i + rows, 0:1] - s[None, :, 0], t[i:i + rows, 1:2] - s[None, :, 1])
        K = torch.complex(-0.25 * torch.special.bessel_y0(r), 0.25 * torch.special.bessel_j0(r))
        out[i:i + rows] = K @ x
    return out


def _dense_system(pts, nrm, w, off, k):
    """1/2 I + (alpha S + beta D + C) diag(w), alpha = -i k, beta = 1, C the
    order-6 Kapur-Rokhlin correction inside every circle."""
    p, nr = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()

    def value(tx, ty, sx, sy, nx, ny):
        dx, dy = tx - sx, ty - sy
        r = torch.hypot(dx, dy)
        zero = r == 0
        r = torch.where(zero, torch.ones_like(r), r)
        S = torch.complex(-0.25 * torch.special.bessel_y0(k * r), 0.25 * torch.special.bessel_j0(k * r))
        f = 0.25 * k / r * (nx * dx + ny * dy)
        D = torch.complex(-f * torch.special.bessel_y1(k * r), f * torch.special.bessel_j1(k * r))
        v = -1j * k * S + D
        return torch.where(zero, torch.zeros_like(v), v)

    n = len(pts)
    A = torch.empty((n, n), dtype=torch.complex128, device="cuda")
    for i in range(0, n, 2048):
        A[i:i + 2048] = value(p[i:i + 2048, 0:1], p[i:i + 2048, 1:2], p[None, :, 0], p[None, :, 1],
                              nr[None, :, 0], nr[None, :, 1])
    i = torch.arange(n, device="cuda")
    curve = torch.bucketize(i, torch.from_numpy(off[1:]).cuda(), right=True)
    i0 = torch.from_numpy(off[:-1]).cuda()[curve]
    m = torch.from_numpy(np.diff(off)).cuda()[curve]
    for q, kw in enumerate(KR6):
        for j in ((i - i0 + q + 1) % m + i0, (i - i0 + m - q - 1) % m + i0):
            A[i, j] += kw * value(p[j, 0], p[j, 1], p[i, 0], p[i, 1], nr[i, 0], nr[i, 1])
    A *= torch.from_numpy(w).cuda()[None, :]
    A[i, i] += 0.5
    return A


def exact(case, seed):
    if case["kind"] == "solve":
        pts, nrm, w, off, b = _scattering(case, seed)
        return torch.linalg.solve(_dense_system(pts, nrm, w, off, case["k"]), b)
    problems = _problems(case, seed)
    n = sum(len(s) for s, _, _ in problems)
    x = _rhs(n, case["rhs"], case["precision"], seed).to(torch.complex128).reshape(n, -1)
    tree = case["kind"] == "apply" and not case["original"]
    if tree:
        sp, tp = _tree_orders(case, problems)
        tree_x, x = x, torch.empty_like(x)
        x[sp] = tree_x
    out, base = [], 0
    for src, tgt, k in problems:
        out.append(_dense_apply(src, tgt, k, x[base:base + len(src)]))
        base += len(src)
    y = torch.cat(out)
    if tree:
        y = y[tp]
    y = y[:, 0] if case["rhs"] == 1 else y
    return y.cpu().numpy() if case["kind"] == "apply" and case["host"] else y

"""A double-float apply of many right-hand sides, which runs on the FP64
factors, makes no copy of them: the pipelined host apply prepares a precision
before each call."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import butterfly_gb300 as B  # noqa: E402


def test_many_right_hand_sides_copy_no_factors():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = B.default_context(0)
    n, R = 12000, 6
    fac = B.FacHelm2.make_multilevel(
        B.Helm2(n / 128.0), B.Quadtree(B.uniform_square_points(n, 2), leaf_size=64),
        B.Quadtree(B.curve_points("ellipse", n), leaf_size=64), rank_eps=1e-10, pinv_tol=1e-10,
        context=ctx)
    X = torch.from_numpy(B.Rng(1).complex_randn(n * R).reshape(n, R)).pin_memory()
    Y = torch.empty_like(X).pin_memory()
    lib, prec = B.lib(), B.PRECISIONS

    def call(name):
        ctx.check(lib.bfgFacApplyHostAsync(fac.handle, prec[name], B._VP(X.data_ptr()), R, R,
                                           B._VP(Y.data_ptr()), R, ctypes.c_uint32(0)))
        ctx.check(lib.bfgFacApplyHostWait(fac.handle))
        return Y.clone()

    a, b = call("fp64"), call("fp64")   # both staging slots, the workspace
    free = torch.cuda.mem_get_info()[0]
    c = call("df64")
    assert free - torch.cuda.mem_get_info()[0] < 8 * fac.stats()["arenaEntries"]
    assert torch.equal(a, b) and torch.equal(a, c)

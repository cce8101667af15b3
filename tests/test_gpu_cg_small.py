"""The one-launch CG of small systems: same iterations, residuals and x to the
bit as the loop of separate launches (loop_mode 2), without a preconditioner
and with the diagonal one, FP64 and FP32, for row counts at the edges of a
tile and of the rows-per-thread choices, and beyond them (where the loop of
launches runs in both modes)."""
import io

import numpy as np
import pytest

from mtl4_b200 import problems as P

pytestmark = pytest.mark.gpu

GRIDS = [(1, 2), (15, 17), (16, 16), (257, 1), (64, 65), (256, 256), (300, 401), (500, 499), (900, 900)]


def run(ctx, A, dtype, kind, mode, iters):
    from mtl4_b200 import itl, mtl
    Ad = mtl.compressed2D.from_problem(A, ctx)
    b = mtl.dense_vector(P.random_rhs(A.n_rows, 3).astype(dtype), dtype, ctx)
    x = mtl.dense_vector(A.n_rows, dtype, ctx)
    Pc = getattr(itl.pc, kind)(Ad, dtype)
    out = io.StringIO()
    it = itl.cyclic_iteration(b, iters, 1e-6, 0.0, 1, out)
    old = ctx.get_tuning("loop_mode")
    ctx.set_tuning("loop_mode", mode)
    try:
        before = ctx.kernel_launches()
        itl.cg(Ad, x, b, Pc, it)
        return x.numpy(), it.iterations(), it.error, it.resid(), out.getvalue(), ctx.kernel_launches() - before
    finally:
        ctx.set_tuning("loop_mode", old)


@pytest.mark.parametrize("shape", GRIDS, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", ["identity", "diagonal"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_one_launch_equals_the_loop_of_launches(ctx, shape, kind, dtype):
    A = P.vardiff_2d(shape, sigma=0.5, seed=6)
    for iters in (0, 1, 2, 31):
        one, many = (run(ctx, A, dtype, kind, mode, iters) for mode in (0, 2))
        assert np.array_equal(one[0], many[0])
        assert one[1:5] == many[1:5]
        if A.n_rows <= 148 * 4 * 256:   # within the smallest range the choice covers on this GPU
            assert one[5] <= 8


def test_refinement_and_repeated_solves(ctx):
    from mtl4_b200 import itl, mtl
    A = P.vardiff_3d((30, 21, 17), sigma=0.7, seed=2)
    Ad = mtl.compressed2D.from_problem(A, ctx)
    got = []
    for mode in (0, 2, 0):
        old = ctx.get_tuning("loop_mode")
        ctx.set_tuning("loop_mode", mode)
        try:
            for seed in (1, 2):
                b = mtl.dense_vector(P.random_rhs(A.n_rows, seed), np.float64, ctx)
                x = mtl.dense_vector(A.n_rows, np.float64, ctx)
                it = itl.refine("cg", Ad, x, b, itl.pc.diagonal(Ad, np.float32))
                got.append((seed, it.iterations(), it.outer, x.numpy()))
        finally:
            ctx.set_tuning("loop_mode", old)
    for a in got[2:]:
        b = got[a[0] - 1]
        assert a[1:3] == b[1:3] and np.array_equal(a[3], b[3])

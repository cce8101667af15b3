"""Waits of the grid sweeps that run out where nobody looks at once: inside a
refinement that goes on, and in queued applies.  The rows half handed over
between tiles belong to the preconditioner, so the next user of it has to
learn of the expiry; afterwards everything is the bits of before."""
import contextlib

import numpy as np
import pytest

from mtl4_b200 import problems as P

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def tuning(ctx, **kv):
    old = {k: ctx.get_tuning(k) for k in kv}
    try:
        for k, v in kv.items():
            ctx.set_tuning(k, v)
        yield
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)


def nearly_identity(shape):
    """A grid operator whose off-diagonal entries hardly matter, so that an
    inner solve on stale neighbours still gains."""
    A = P.vardiff_3d(shape, sigma=0.2, seed=4, beta=(0.2, 0.1, 0.05))
    rows = np.repeat(np.arange(A.n_rows), np.diff(A.row_ptr))
    A.val[:] = np.where(rows == A.col, 1.0, 1e-9 * A.val / np.abs(A.val).max())
    return A


def test_refinement_stops_at_the_inner_loop_whose_wait_ran_out(ctx):
    from mtl4_b200 import _lib, itl, mtl
    A = nearly_identity((40, 36, 33))
    Ad = mtl.compressed2D.from_problem(A, ctx)
    b = mtl.dense_vector(P.random_rhs(A.n_rows, 1), np.float64, ctx)

    def refine(Pc, outer):
        x = mtl.dense_vector(A.n_rows, np.float64, ctx)
        before = ctx.kernel_launches()
        try:
            itl.refine("bicgstab", Ad, x, b, Pc, rtol=1e-300, inner_rtol=1e-30, max_outer=outer, max_inner=1)
            expired = False
        except _lib.device_timeout:
            expired = True
        return expired, ctx.kernel_launches() - before, x.numpy()

    Pc = itl.pc.ilu_0(Ad, np.float32)
    assert Pc.sweep_plan(np.float32)["kernel"] == "grid"
    expired, one_outer, _ = refine(Pc, 1)
    assert not expired
    v = mtl.dense_vector(P.random_rhs(A.n_rows, 2).astype(np.float32), np.float32, ctx)
    want = itl.solve(Pc, v).numpy()
    Pw = itl.pc.ilu_0(Ad, np.float32)   # a set's limit is the one of its first solve
    with tuning(ctx, spin_limit=1):
        expired, launches, _ = refine(Pw, 8)
    assert expired and launches <= one_outer
    assert np.array_equal(itl.solve(Pw, v).numpy(), want)


@pytest.mark.parametrize("solver", ["bicgstab", "refine"])
def test_queued_apply_that_ran_out_is_reported_by_a_solve(ctx, solver):
    from mtl4_b200 import _lib, itl, mtl
    A = P.convdiff_3d(32)
    st = np.float32 if solver == "refine" else np.float64
    Ad = mtl.compressed2D.from_problem(A, ctx)
    Pc = itl.pc.ilu_0(Ad, st)
    b = mtl.dense_vector(P.random_rhs(A.n_rows, 1), np.float64, ctx)
    v, y = mtl.dense_vector(P.random_rhs(A.n_rows, 2).astype(st), st, ctx), mtl.dense_vector(A.n_rows, st, ctx)

    def solve():
        x = mtl.dense_vector(A.n_rows, np.float64, ctx)
        if solver == "refine":
            it = itl.refine("bicgstab", Ad, x, b, Pc)
        else:
            it = itl.basic_iteration(b, 500, 1e-8)
            itl.bicgstab(Ad, x, b, Pc, it)
        return it.iterations(), x.numpy()

    n0, x0 = solve()
    with tuning(ctx, pc_apply_sync=0):
        itl.solve(Pc, v, y)
        assert solve()[0] == n0   # queued applies that ran through
        with tuning(ctx, spin_limit=1):
            itl.solve(Pc, v, y)
    with pytest.raises(_lib.device_timeout):
        solve()
    for _ in range(2):
        n1, x1 = solve()
        assert n1 == n0 and np.array_equal(x1, x0)

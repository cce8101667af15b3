"""Grid sweeps at the edges of their tiles: lines shorter and longer than a
warp's skew, a staged block and the rings; sides one below, at and one above
a warp's 8 x 4 (or 32) lines and a tile's 16 x 8 (or 128) lines; several
tiles in both directions.  The applies are the oracle's bit for bit (the same
arithmetic per row in another schedule), repeated so that rings, hand-off
rows and counts are seen to come back to their start state."""
import numpy as np
import pytest

from mtl4_b200 import problems as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (2, 9, 5), (5, 8, 4), (7, 16, 8), (8, 17, 9), (9, 7, 33), (40, 33, 3), (33, 15, 17),
          (3, 31), (8, 32), (9, 33), (70, 127), (31, 128), (5, 129), (64, 300)]


def build(shape):
    f = P.vardiff_3d if len(shape) == 3 else P.vardiff_2d
    return f(shape, sigma=0.5, seed=11, beta=(0.2, 0.1, 0.05)[:len(shape)])


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_applies_at_tile_edges(ctx, shape):
    from mtl4_b200 import itl, mtl
    A = build(shape)
    Ad = mtl.compressed2D.from_problem(A, ctx)
    x = np.random.default_rng(3).standard_normal(A.n_rows)
    old = ctx.get_tuning("grid_warps")
    try:
        for warps in (4, 8):
            ctx.set_tuning("grid_warps", warps)
            for kind in ("ilu_0", "ic_0"):
                for st, vt in ((np.float64, np.float64), (np.float32, np.float32), (np.float32, np.float64)):
                    Pc = getattr(itl.pc, kind)(Ad, st)
                    assert Pc.sweep_plan(vt)["kernel"] == "grid"
                    want = (O.port_pc_apply(A, kind, x.astype(np.float32)) if vt == np.float32
                            else O.port_pc_apply(A, kind, x, storage_f32=(st == np.float32)))
                    xv = mtl.dense_vector(x.astype(vt), vt, ctx)
                    for _ in range(2):
                        assert np.array_equal(itl.solve(Pc, xv).numpy(), want), (kind, st, vt, warps)
    finally:
        ctx.set_tuning("grid_warps", old)


def test_grid_and_flat_sweeps_in_turn(ctx):
    # grid sweeps leave values in the vector between the two sweeps, which a
    # flat sweep of the same preconditioner wants all sentinel
    from mtl4_b200 import itl, mtl
    A = build((20, 18, 11))
    Pc = itl.pc.ilu_0(mtl.compressed2D.from_problem(A, ctx))
    x = np.random.default_rng(4).standard_normal(A.n_rows)
    want = O.port_pc_apply(A, "ilu_0", x)
    xv = mtl.dense_vector(x, np.float64, ctx)
    old = ctx.get_tuning("sweep_kernel")
    try:
        for k in (0, 1, 0, 1, 1, 0):
            ctx.set_tuning("sweep_kernel", k)
            assert np.array_equal(itl.solve(Pc, xv).numpy(), want)
    finally:
        ctx.set_tuning("sweep_kernel", old)

"""The limit of the grid sweeps' waits is one wait's: a tile's receiver warps
come by their rows in thousands of polls over long lines, of which each brings
some, and may use the limit up for none of them.  The back-off between polls
("sweep_sleep_ns") changes no result."""
import numpy as np
import pytest

from mtl4_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape", [(20000, 130), (20000, 9, 17)], ids=lambda s: "x".join(map(str, s)))
def test_long_lines_do_not_use_up_the_limit(ctx, shape, dtype):
    from mtl4_b200 import itl, mtl
    # several tiles, lines of 20,000 rows
    A = (P.vardiff_3d if len(shape) == 3 else P.vardiff_2d)(shape, sigma=0.2, seed=4)
    Pc = itl.pc.ilu_0(mtl.compressed2D.from_problem(A, ctx), dtype)
    assert Pc.sweep_plan(dtype)["kernel"] == "grid"
    x = mtl.dense_vector(np.random.default_rng(1).standard_normal(A.n_rows), dtype, ctx)
    want = itl.solve(Pc, x).numpy()
    old = {k: ctx.get_tuning(k) for k in ("spin_limit", "sweep_sleep_ns")}
    try:
        ctx.set_tuning("spin_limit", 1000)
        for _ in range(3):
            assert np.array_equal(itl.solve(Pc, x).numpy(), want)
        ctx.set_tuning("sweep_sleep_ns", 400)
        assert np.array_equal(itl.solve(Pc, x).numpy(), want)
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)

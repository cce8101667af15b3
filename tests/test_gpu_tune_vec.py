"""The vector passes' launch shape is chosen by timing those passes, also on
systems small enough for the one-launch CG, which has none."""
import numpy as np
import pytest

from mtl4_b200 import autotune, problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [40, 200])
def test_every_candidate_runs_the_vector_passes(ctx, m, tmp_path):
    from mtl4_b200 import mtl
    A = P.vardiff_2d(m, sigma=0.3, seed=2)
    Ad = mtl.compressed2D.from_problem(A, ctx)
    old = {k: ctx.get_tuning(k) for k in ("vec_ctas_per_sm", "loop_mode")}
    iters, reps = 30, 2
    try:
        before = ctx.kernel_launches()
        choice, cached = autotune.tune_vec(ctx, Ad, np.float64, autotune.Cache(tmp_path / "c.json"), iters, reps)
        assert not cached and choice["vec_ctas_per_sm"] in autotune.VEC_CTAS
        assert ctx.get_tuning("vec_ctas_per_sm") == choice["vec_ctas_per_sm"]
        assert ctx.get_tuning("loop_mode") == old["loop_mode"]
        # a product and a vector pass per iteration, one warm-up run per candidate
        assert ctx.kernel_launches() - before >= len(autotune.VEC_CTAS) * (reps + 1) * 2 * iters
    finally:
        for k, v in old.items():
            ctx.set_tuning(k, v)

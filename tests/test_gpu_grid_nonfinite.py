"""Infinities and NaN through the grid sweeps.  Outside the grid and past a
line's ends the kernel multiplies padding (+0) by whatever a neighbouring lane
holds and takes no validity tests, so a value that is not finite must not get
into rows that do not depend on it: every element is the oracle's, NaN where
it has NaN."""
import numpy as np
import pytest

from mtl4_b200 import problems as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# several tiles, lines of odd lengths, off lanes in the last units
SHAPES = [(9, 19, 11), (33, 17, 9), (5, 40, 3), (40, 133), (7, 300)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", ["ilu_0", "ic_0"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_applies_with_values_that_are_not_finite(ctx, shape, kind, dtype):
    from mtl4_b200 import itl, mtl
    A = (P.vardiff_3d if len(shape) == 3 else P.vardiff_2d)(shape, sigma=0.5, seed=11)
    Pc = getattr(itl.pc, kind)(mtl.compressed2D.from_problem(A, ctx), dtype)
    assert Pc.sweep_plan(dtype)["kernel"] == "grid"
    n, nx = A.n_rows, shape[0]
    clean = np.random.default_rng(3).standard_normal(n).astype(dtype)
    # ends of lines, the first and the last row, the middle
    for at in (0, nx - 1, nx, n // 2, n - nx, n - 1):
        for v in (np.inf, -np.inf, np.nan, np.finfo(dtype).max, np.finfo(dtype).min):
            x = clean.copy()
            x[at] = v
            with np.errstate(all="ignore"):
                want = O.port_pc_apply(A, kind, x)
            got = itl.solve(Pc, mtl.dense_vector(x, dtype, ctx)).numpy()
            assert np.array_equal(got, want, equal_nan=True), (at, v)
    # the next apply is untouched by the hand-off rows of those before
    assert np.array_equal(itl.solve(Pc, mtl.dense_vector(clean, dtype, ctx)).numpy(), O.port_pc_apply(A, kind, clean))

"""Which systems the one-launch CG takes: not those whose product tiles are not
whole 256-row tiles (2048 entries fill a tile first: 9-point operators), where
its sums would be other ones than the loop's."""
import numpy as np
import pytest

from mtl4_b200.problems import CSR

pytestmark = pytest.mark.gpu


def nine_point(nx, ny):
    """Symmetric 9-point operator, diagonally dominant, in row order."""
    k = np.exp(0.3 * np.random.default_rng(nx * ny).standard_normal((ny, nx)))
    rows, cols, vals = [], [], []
    for j in range(ny):
        for i in range(nx):
            row = {}
            for dj in (-1, 0, 1):
                for di in (-1, 0, 1):
                    if (di or dj) and 0 <= i + di < nx and 0 <= j + dj < ny:
                        row[(j + dj) * nx + i + di] = -k[j, i] * k[j + dj, i + di] / (1 + abs(di) + abs(dj))
            row[j * nx + i] = 0.05 - sum(row.values())
            cols += sorted(row)
            vals += [row[c] for c in sorted(row)]
            rows.append(len(row))
    rp = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    return CSR(nx * ny, nx * ny, rp, np.asarray(cols, np.int32), np.asarray(vals))


def run(ctx, A, dtype, kind, mode, iters):
    from mtl4_b200 import itl, mtl
    Ad = mtl.compressed2D.from_problem(A, ctx)
    b = mtl.dense_vector(np.random.default_rng(3).standard_normal(A.n_rows).astype(dtype), dtype, ctx)
    x = mtl.dense_vector(A.n_rows, dtype, ctx)
    it = itl.basic_iteration(b, iters, 1e-6)
    old = ctx.get_tuning("loop_mode")
    ctx.set_tuning("loop_mode", mode)
    try:
        itl.cg(Ad, x, b, getattr(itl.pc, kind)(Ad, dtype), it)
    finally:
        ctx.set_tuning("loop_mode", old)
    return x.numpy(), it.iterations(), it.error, it.resid()


# 20 x 20 (242 + 158 rows) and 24 x 25 (three tiles) have as many tiles as
# whole ones would make; 16 x 16 and 40 x 40 do not; 3 x 80 fits one whole tile
@pytest.mark.parametrize("shape", [(20, 20), (24, 25), (16, 16), (40, 40), (3, 80)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", ["identity", "diagonal"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_sums_are_those_of_the_loop_of_launches(ctx, shape, kind, dtype):
    A = nine_point(*shape)
    for iters in (1, 31):
        one, many = (run(ctx, A, dtype, kind, mode, iters) for mode in (0, 2))
        assert np.array_equal(one[0], many[0])
        assert one[1:] == many[1:]

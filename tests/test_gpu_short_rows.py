"""Products of short regular rows inside solves (thread per row) and the
vector passes' grouped dots: the results are those of the staged-tile
product to the bit, for rows of up to eight entries and more, row counts
around a tile (256) and around the tiles whose sums wait together (32 x 256),
and for sets that mix systems; dots equal a restatement of the reduction."""
import numpy as np
import pytest

from mtl4_b200 import problems as P

pytestmark = pytest.mark.gpu


def tile_dot(x, y):
    """Sum of x*y as the device adds it: per 256-row tile a warp tree and a
    tree over the warps, then tiles t, t + 256, ... per thread and the same
    trees over the threads."""
    def tree(v):   # v: [..., 256]
        w = v.reshape(v.shape[:-1] + (8, 32))
        for o in (16, 8, 4, 2, 1):
            w = w[..., :o] + w[..., o:2 * o]
        t = w[..., 0] + 0.0
        for o in (4, 2, 1):
            t = t[..., :o] + t[..., o:2 * o]
        return t[..., 0]
    n = x.size
    pad = (-n) % 256
    p = tree(np.pad(x * y, (0, pad)).reshape(-1, 256))
    acc = np.zeros(256)
    for a in range(0, p.size, 256):
        q = p[a:a + 256]
        acc[:q.size] += q
    return float(tree(acc))


@pytest.mark.parametrize("n", [1, 255, 256, 257, 8191, 8192, 8193, 70001])
def test_dot_order(ctx, n):
    from mtl4_b200 import mtl
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    xd, yd = mtl.dense_vector(x, np.float64, ctx), mtl.dense_vector(y, np.float64, ctx)
    assert mtl.dot(xd, yd) == tile_dot(x, y)
    assert mtl.two_norm(xd) == np.sqrt(tile_dot(x, x))


def banded(n, width):
    offs = np.arange(-(width // 2), width - width // 2)
    r, c = [], []
    for o in offs:
        i = np.arange(max(0, -o), min(n, n - o))
        r.append(i)
        c.append(i + o)
    r, c = np.concatenate(r), np.concatenate(c)
    rng = np.random.default_rng(5)
    v = -rng.random(r.size)
    v[r == c] = width + 1.0
    return P._from_coo(n, r, c, v)


@pytest.mark.parametrize("n,width", [(100, 3), (256, 8), (257, 9), (2000, 12), (8449, 5)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_product_with_dot_equals_staged_tiles(ctx, n, width, dtype):
    from mtl4_b200 import mtl
    A = mtl.compressed2D.from_problem(banded(n, width), ctx)
    x = mtl.dense_vector(np.random.default_rng(2).standard_normal(n).astype(dtype), dtype, ctx)
    got = []
    old = ctx.get_tuning("spmv_kernel")
    try:
        for k in (0, 1):   # automatic (short rows), stream tiles
            ctx.set_tuning("spmv_kernel", k)
            y = mtl.dense_vector(n, dtype, ctx)
            got.append((mtl.mult_dot(A, x, y), y.numpy()))
    finally:
        ctx.set_tuning("spmv_kernel", old)
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])


def test_mixed_set_equals_systems_alone(ctx):
    # short-row systems of several sizes in one set, and a set that a system
    # of longer rows keeps on staged tiles: each system's solve is its own
    from mtl4_b200 import serve
    short = [P.vardiff_2d((37, 21), sigma=0.5, seed=1), P.vardiff_3d((9, 8, 7), sigma=0.5, seed=2), banded(300, 7)]
    long = [banded(400, 25)]

    def solve(As):
        B = serve.batch(ctx)
        for k, A in enumerate(As):
            B.add(A, P.random_rhs(A.n_rows, 7 + A.n_rows), "cg", "ic_0", max_iter=500, rtol=1e-9)
        B.solve()
        return [B.result(i) for i in range(len(As))]

    alone = [solve([A])[0] for A in short]
    for together in (solve(short), solve(short + long)):
        for a, b in zip(alone, together):
            # (the unsymmetric one runs out of iterations, alone as in the set)
            assert a.error_code == b.error_code and a.iterations == b.iterations and np.array_equal(a.x, b.x)

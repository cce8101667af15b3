"""Where the in-solve product changes between a thread per row and staged
tiles (mean row lengths of 7, 9 and 12 entries; between two and three tiles
per SM): the solves are the same bits as in a set whose other system's long
rows make every product a staged one."""
import numpy as np
import pytest

from mtl4_b200.problems import CSR

pytestmark = pytest.mark.gpu


def banded(n, width, seed):
    """Diagonally dominant band of `width` entries a row (fewer at the ends)."""
    rng = np.random.default_rng(seed)
    offs = np.arange(-(width // 2), width - width // 2)
    cols = np.arange(n)[:, None] + offs[None, :]
    inside = (cols >= 0) & (cols < n)
    vals = np.where(offs[None, :] == 0, 2.0 + width, rng.standard_normal((n, width)))
    rp = np.concatenate([[0], np.cumsum(inside.sum(1))]).astype(np.int64)
    return CSR(n, n, rp, cols[inside].astype(np.int32), vals[inside])


def long_rows():
    A = banded(60, 41, 1)   # rows of more than 32 entries
    assert np.diff(A.row_ptr).max() > 32
    return A


# rows per tile: 256, or what 2048 entries hold
@pytest.mark.parametrize("solver,width", [("bicgstab", 5), ("bicgstab", 7), ("bicgstab", 8), ("bicgstab", 12),
                                          ("cg", 9), ("cg", 10), ("cg", 12)])
@pytest.mark.parametrize("per_sm", [1, 2, 3])
@pytest.mark.parametrize("beyond", [-40, 40])
def test_solves_across_the_lines(ctx, solver, width, per_sm, beyond):
    from mtl4_b200 import serve
    n = per_sm * ctx.get_tuning("sm_count") * min(256, 2048 // width) + beyond
    A, b = banded(n, width, n), np.random.default_rng(n).standard_normal(n)
    B = long_rows()
    got = []
    for mixed in (False, True):
        for systems in ([A], [A, B]):
            bt = serve.batch(ctx)
            for S in systems:
                bt.add(S, b[:S.n_rows], solver, "identity", max_iter=6, rtol=1e-30)
            bt.solve(mixed=mixed, rtol=1e-30, inner_rtol=1e-30, max_outer=1, max_inner=6)
            got.append((bt.result(0).x, bt.result(0).iterations))
            del bt
    for alone, together in (got[:2], got[2:]):
        assert alone[1] == together[1] and np.array_equal(alone[0], together[0])

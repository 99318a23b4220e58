"""Triangular solves at the edges of a group of 8 right-hand sides, of the rule
for narrow products (32) and of the 64-column tiles: two fronts whose column
and row counts lie around the 64-row tiles and the 128-deep chunks, both
triangles, static and dynamic order, atomic and ordered sums, against dense
solves with the same factor."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import grids

pytestmark = pytest.mark.gpu


def dense_factor(nn, na, extra):
    """A two-front pattern, its factor on the GPU and dense in reordered numbering."""
    n = nn + na + extra
    r, c = np.tril_indices(n, -1)
    keep = (c >= nn) | (r < nn + na)
    A = grids.spd_from_lower_pattern(n, r[keep], c[keep], nn + 100 * na)
    s = cp.symbolic(A)
    assert [int(x) for x in np.diff(s.snptr)] == [nn, na + extra]
    X = cp.cspmatrix(s) + A
    cp.cholesky(X)
    v = X.blkval.cpu().numpy()
    L = np.zeros((n, n))
    for k in range(s.Nsn):
        j0, j1 = int(s.snptr[k]), int(s.snptr[k + 1])
        rows = np.asarray(s.snrowidx[int(s.sncolptr[k]):int(s.sncolptr[k + 1])]).reshape(-1)
        b = v[int(s.blkptr[k]):int(s.blkptr[k + 1])].reshape(j1 - j0, len(rows)).T
        # (the rows below a diagonal block are stored times its inverse)
        D = np.tril(b[:j1 - j0])
        L[np.ix_(rows, np.arange(j0, j1))] = np.vstack([D, b[j1 - j0:] @ D])
    return s, X, L


@pytest.mark.parametrize("nn,na,extra", [(3, 0, 2), (5, 7, 1), (64, 63, 3), (65, 130, 3), (129, 64, 130), (320, 65, 200)])
@pytest.mark.parametrize("mode,ordered", [("static", 0), ("dynamic", 0), ("static", 1)])
def test_solves(nn, na, extra, mode, ordered):
    s, X, L = dense_factor(nn, na, extra)
    plan = s.plan(0)
    plan.set_schedule(mode)
    plan.set_option("ordered_sums", ordered)
    p = np.asarray(s.p).reshape(-1)
    n = s.n
    # solving by blocks of 64 rows with their inverses, precomputed products
    # with them and sums in any order, each is wrong by at most
    # n eps |L^-1| |L| |L^-1| |L| |x|; with the dense solve's own, 4 of them
    Li = np.abs(np.linalg.inv(L))
    G = 4 * n * 2.0**-53 * (Li @ np.abs(L) @ Li @ np.abs(L))
    for nrhs in (1, 7, 8, 9, 32, 33, 65):
        B = np.random.default_rng(nrhs).standard_normal((n, nrhs))
        for trans in "NT":
            Bg = torch.from_numpy(B.T.copy()).cuda().t()
            cp.trsm(X, Bg, trans=trans)
            want = np.linalg.solve(L if trans == "N" else L.T, B[p])
            Gt = G if trans == "N" else 4 * n * 2.0**-53 * (Li.T @ np.abs(L).T @ Li.T @ np.abs(L).T)
            assert np.all(np.abs(Bg.cpu().numpy()[p] - want) <= Gt @ np.abs(want) + 1e-300), (nrhs, trans)

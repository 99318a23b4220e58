"""Backward errors of cholesky on small fronts whose pivot block is
ill-conditioned: the factor and the rows below it, componentwise, for fronts
of their own task (bundles off) and for bundles; the rounding and the range of
a bundle's pivots; a value that is not finite in projected_inverse."""
import numpy as np
import pytest
import torch

import chompack_b200 as cp
from chompack_b200 import grids

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
EXTRA = 3


def kahan(n, rng, angle):
    c, s = np.cos(angle), np.sin(angle)
    return (np.eye(n) - c * np.tril(np.ones((n, n)), -1)) * s ** (np.arange(n) % 16) * (1 + 0.1 * rng.random((n, n)))


def front(nn, na, seed):
    """Block values of a front of nn columns and na rows below them, under a
    root of na + EXTRA columns; A11 = L11 L11^T with L11 ill-conditioned."""
    rng = np.random.default_rng(seed)
    L = kahan(nn, rng, 1.0 if nn <= 24 else 1.25).astype(np.longdouble)
    W = rng.standard_normal((na, nn)).astype(np.longdouble)
    A11 = (L @ L.T).astype(np.float64)
    A21 = (W @ L @ L.T).astype(np.float64)
    nr = na + EXTRA
    R = np.tril(rng.standard_normal((nr, nr))) + 3 * np.eye(nr)
    A22 = R @ R.T
    A22[:na, :na] += ((W @ L) @ (W @ L).T).astype(np.float64)
    return A11, A21, A22


@pytest.mark.parametrize("bundles", [0, 1])
@pytest.mark.parametrize("nn,na", [(3, 20), (5, 11), (9, 20), (16, 16), (16, 40), (24, 33), (33, 31), (47, 17)])
def test_backward_error(nn, na, bundles):
    if bundles and nn + na > 32:
        pytest.skip("bundles hold fronts of at most 32 rows")
    n = nn + na + EXTRA
    r, c = np.tril_indices(n, -1)
    keep = (c >= nn) | (r < nn + na)
    s = cp.symbolic(grids.spd_from_lower_pattern(n, r[keep], c[keep], 0))
    assert [int(x) for x in np.diff(s.snptr)] == [nn, na + EXTRA]
    s.plan().set_option("subtrees", bundles)
    A11, A21, A22 = front(nn, na, 10 * nn + na)
    x = np.concatenate([np.concatenate([np.tril(A11), A21]).ravel(order="F"), np.tril(A22).ravel(order="F")])
    X = cp.cspmatrix(s, blkval=torch.from_numpy(x).cuda())
    cp.cholesky(X)
    got = X.blkval.cpu().numpy()[:(nn + na) * nn].reshape(nn, nn + na).T.astype(np.longdouble)
    L, W = np.tril(got[:nn]), got[nn:]
    # |A11 - L L^T| <= gamma_(nn + 1) |L| |L^T|, and a few roundings for the
    # reciprocals; W solves X L^T = A21, then W L = X, each within gamma_nn
    g = (nn + 4) * U
    aL = np.abs(L)
    assert np.all(np.abs(A11 - L @ L.T) <= g * (aL @ aL.T))
    assert np.all(np.abs(A21 - W @ (L @ L.T)) <= 2.1 * g * (np.abs(W) @ (aL @ aL.T)))


def test_bundle_pivots():
    # leaves of one column under a root of four (the last leaf is in the root)
    m, nr = 301, 4
    r = np.concatenate([np.tile(np.arange(m, m + nr), m), m + np.tril_indices(nr, -1)[0]])
    c = np.concatenate([np.repeat(np.arange(m), nr), m + np.tril_indices(nr, -1)[1]])
    s = cp.symbolic(grids.spd_from_lower_pattern(m + nr, r, c, 0))
    nn = np.diff(s.snptr)
    assert s.Nsn == m and np.count_nonzero(nn == 1) == m - 1
    rng = np.random.default_rng(1)
    x = np.zeros(int(s.blkptr[-1]))
    at = np.array([int(s.blkptr[k]) for k in range(m) if nn[k] == 1])
    x[at] = rng.uniform(1.0, 4.0, m - 1)
    x[at[:, None] + np.arange(1, nr + 1)] = rng.standard_normal((m - 1, nr))
    k = int(np.argmax(nn))
    root = slice(int(s.blkptr[k]), int(s.blkptr[k + 1]))
    x[root][::nr + 2] = 10.0 * m

    def factor(v):
        X = cp.cspmatrix(s, blkval=torch.from_numpy(v.copy()).cuda())
        cp.cholesky(X)
        return X.blkval.cpu().numpy()

    L = factor(x)
    assert np.array_equal(L[at], np.sqrt(x[at]))
    # an infinite pivot: its column vanishes, the other leaves stay as they are
    x[at[7]] = np.inf
    Li = factor(x)
    assert Li[at[7]] == np.inf and not np.any(Li[at[7] + 1:at[7] + 1 + nr])
    other = np.delete(at, 7)[:, None] + np.arange(nr + 1)
    assert np.array_equal(Li[other], L[other]) and np.all(np.isfinite(Li[root]))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n,row,col", [(20, 17, 3), (40, 20, 3), (40, 39, 17), (64, 50, 30), (33, 32, 0)])
def test_non_finite_entry_stays_in_its_columns(n, row, col, value):
    # one front; Y(i, j) depends on L(row, col) only where min(i, j) <= col
    A = grids.random_lower(n, 1.0, seed=n)
    s = cp.symbolic(A)
    assert s.Nsn == 1
    s.plan().set_option("subtrees", 0)
    M = (cp.cspmatrix(s, device="cpu") + A).blkval.numpy().reshape(n, n, order="F")
    L = np.linalg.cholesky(np.tril(M) + np.tril(M, -1).T)
    T = np.linalg.inv(L[col + 1:, col + 1:])
    L[row, col] = value
    X = cp.cspmatrix(s, blkval=torch.from_numpy(L.ravel(order="F").copy()).cuda(), factor=True)
    cp.projected_inverse(X)
    Y = X.blkval.cpu().numpy().reshape(n, n, order="F")[col + 1:, col + 1:]
    want = np.tril(T.T @ T)
    assert np.all(np.abs(np.tril(Y) - want) <= 1e-13 * np.abs(want).max())


def fma(a, b, c):
    return (np.asarray(a, np.longdouble) * b + c).astype(np.float64)


def scalar_inverse(L):
    """(L L^T)^{-1} as an unblocked inverse from the last column to the first
    and sequential dots give it in double precision."""
    n = len(L)
    M, Y = L.copy(), np.zeros((n, n))
    for j in range(n - 1, -1, -1):
        a, t = 1.0 / M[j, j], np.zeros(n)
        for k in range(j + 1, n):
            t[k:] = fma(M[k:, k], M[k, j], t[k:])
        M[j + 1:, j], M[j, j] = -a * t[j + 1:], a
    for k in range(n):
        Y = fma(M[k][:, None], M[k][None, :], Y)
    return Y


@pytest.mark.parametrize("n,decades", [(40, 6), (40, 10), (64, 10)])
def test_inverse_is_as_exact_as_a_scalar_one(n, decades):
    # 40 rotated spectra, one blocked front each; the two errors are those of
    # two rounding sequences of one size, so their mean log ratio is within
    # three standard errors of zero
    s = cp.symbolic(grids.random_lower(n, 1.0, seed=n))
    s.plan().set_option("subtrees", 0)
    here, scalar = [], []
    for seed in range(40):
        Q = np.linalg.qr(np.random.default_rng(seed).standard_normal((n, n)))[0]
        A = (Q * 10.0 ** np.linspace(0, -decades, n)) @ Q.T
        L = np.linalg.cholesky((A + A.T) / 2)
        T = np.eye(n, dtype=np.longdouble)
        for i in range(n):
            T[i] = (T[i] - L[i, :i] @ T[:i]) / L[i, i]
        want = np.tril(T.T @ T)
        X = cp.cspmatrix(s, blkval=torch.from_numpy(L.ravel(order="F").copy()).cuda(), factor=True)
        cp.projected_inverse(X)
        for e, Y in ((here, X.blkval.cpu().numpy().reshape(n, n, order="F")), (scalar, scalar_inverse(L))):
            d = np.tril(Y) - want
            e.append(float(np.sqrt(np.sum(d * d) / np.sum(want * want))))
    ratio = np.log(np.array(here) / np.array(scalar))
    assert ratio.mean() <= 3.0 * ratio.std(ddof=1) / np.sqrt(len(ratio)), (ratio.mean(), ratio.std())


@pytest.mark.parametrize("nn,na", [(8, 24), (16, 40), (40, 20)])
def test_inverse_with_rows_below_is_as_exact_as_a_scalar_one(nn, na):
    # a front under a root: Y21 = -V W, Y11 = M^T M - Y21^T W with V out of the
    # root's result; 40 diagonally dominant matrices, compared as above
    n = nn + na + EXTRA
    r, c = np.tril_indices(n, -1)
    keep = (c >= nn) | (r < nn + na)
    pattern = [grids.spd_from_lower_pattern(n, r[keep], c[keep], seed) for seed in range(40)]
    s = cp.symbolic(pattern[0])
    s.plan().set_option("subtrees", 0)
    here, scalar = [], []
    for A in pattern:
        X = cp.cspmatrix(s) + A
        cp.cholesky(X)
        B = X.blkval.cpu().numpy()[:(nn + na) * nn].reshape(nn, nn + na).T
        L, W = np.tril(B[:nn]), B[nn:]
        cp.projected_inverse(X)
        Y = X.blkval.cpu().numpy()
        V = Y[(nn + na) * nn:].reshape(na + EXTRA, na + EXTRA).T[:na, :na]
        V = np.tril(V) + np.tril(V, -1).T
        T = np.eye(nn, dtype=np.longdouble)
        for i in range(nn):
            T[i] = (T[i] - L[i, :i] @ T[:i]) / L[i, i]
        want = T.T @ T + W.T.astype(np.longdouble) @ (V.astype(np.longdouble) @ W)
        S, P = np.zeros((na, nn)), np.zeros((nn, nn))
        for k in range(na):
            S = fma(V[:, k:k + 1], W[k:k + 1], S)
        for k in range(na):
            P = fma(-S[k][:, None], W[k][None, :], P)
        for e, Z in ((here, Y[:(nn + na) * nn].reshape(nn, nn + na).T[:nn]), (scalar, scalar_inverse(L) - P)):
            d = np.tril(Z) - np.tril(want)
            e.append(float(np.sqrt(np.sum(d * d))))
    ratio = np.log(np.array(here) / np.array(scalar))
    assert ratio.mean() <= 3.0 * ratio.std(ddof=1) / np.sqrt(len(ratio)), (ratio.mean(), ratio.std())

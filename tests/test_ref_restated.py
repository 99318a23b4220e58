"""The oracle without the reference's kernels: every function of oracle/ref.py
answers from the C restatement, and the restated product form satisfies its
definition."""
import numpy as np
import pytest

import golden_cases as G
from helpers import assert_blocks_close
from oracle import ref


@pytest.fixture(autouse=True)
def no_reference_kernels(monkeypatch):
    monkeypatch.setattr(ref, "LIB", "/nonexistent")
    monkeypatch.setattr(ref, "_lib", None)


def test_sweeps():
    d, A, s = G.load("rand200_m164")
    L = d["blkval"].copy()
    assert ref.cholesky(s, L) == 0
    assert_blocks_close(s, L, d["ref_cholesky"])
    r = L.copy()
    assert ref.projected_inverse(s, r) == 0
    assert_blocks_close(s, r, d["ref_projected_inverse"])
    assert ref.completion(s, r, factored_updates=True) == 0
    assert_blocks_close(s, r, d["ref_completion_fu1"])
    B = np.asfortranarray(np.random.default_rng(0).standard_normal((s.n, 3)))
    X = B.copy(order="F")
    ref.trsm(s, L, X, alpha=2.0, trans='N')
    ref.trsm(s, L, X, alpha=0.5, trans='T')
    M = np.zeros((s.n, s.n))
    np.add.at(M, (d["I"].astype(int), d["J"].astype(int)), d["V"])
    M = np.tril(M) + np.tril(M, -1).T
    assert np.max(np.abs(M @ X - B)) <= 1e-11 * np.max(np.abs(B))
    assert "restatement" in ref.source() and not ref.set_threads(2)


@pytest.mark.parametrize("n,k", [(1, 1), (31, 2), (60, 5)])
def test_product_form(n, k):
    rng = np.random.default_rng(n)
    V0 = np.asfortranarray(rng.standard_normal((n, k)))
    a = rng.uniform(0.5, 2.0, k)
    V = V0.copy(order="F")
    L, B, info = ref.pfchol(a, V)
    assert info == 0
    U0 = np.asfortranarray(rng.standard_normal((n, 4)))
    U = ref.pftrmm(V, L, B, ref.pftrmm(V, L, B, U0.copy(order="F"), 'T'), 'N')
    want = U0 + V0 @ (a[:, None] * (V0.T @ U0))
    assert np.max(np.abs(U - want)) <= 1e-11 * np.max(np.abs(want))
    ref.pftrsm(V, L, B, ref.pftrsm(V, L, B, U, 'N'), 'T')
    assert np.max(np.abs(U - U0)) <= 1e-10 * np.max(np.abs(want))
    assert ref.pfchol(-a * n * 100.0, V0 + 1.0)[2] == -1

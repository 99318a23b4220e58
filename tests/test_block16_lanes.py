"""The warp routine of the 16 x 16 diagonal blocks on the CPU (see
block16_lanes.cpp): pivots over the whole range of the type, a failing
pivot, the inverse in place of the block and its residual."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LD = 20
U = 2.0 ** -53


@pytest.fixture(scope="module")
def block16(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("lanes") / "block16.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    "-I", os.path.join(HERE, "..", "chompack_b200", "csrc"), os.path.join(HERE, "block16_lanes.cpp"),
                    "-o", so], check=True)
    fn = ctypes.CDLL(so).block16

    def call(block, factor, cols=16, down=False, in_place=False):
        """(L, M, info) for the lower part of a 16 x 16 block."""
        buf = np.zeros((2, 16, LD))
        buf[0, :, :16] = np.tril(block).T
        p = [buf[i].ctypes.data_as(ctypes.c_void_p) for i in range(2)]
        info = fn(p[0], p[0] if in_place else p[1], int(factor), cols, int(down))
        L, M = buf[0, :, :16].T.copy(), buf[0 if in_place else 1, :, :16].T.copy()
        return L, M, info
    return call


def spd(cols, seed, scale=1.0):
    """A block of `cols` columns in the leading part of a 16 x 16 identity."""
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((cols, cols))
    A = np.eye(16)
    A[:cols, :cols] = (G @ G.T + np.eye(cols)) * scale
    return A


@pytest.mark.parametrize("scale", [1.0, 1e-306, 1e-290, 1e300])
@pytest.mark.parametrize("cols", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("down", [False, True])
def test_factor(block16, cols, scale, down):
    A = spd(cols, cols, scale)
    L, M, info = block16(A, True, cols, down)
    assert info == -1
    # Cholesky's componentwise bound for 16 columns, with a reciprocal square
    # root and a product in place of a square root and divisions
    Ll = np.tril(L[:cols, :cols]).astype(np.longdouble)
    err = np.abs(Ll @ Ll.T - A[:cols, :cols])
    assert np.all(err <= 20 * U * (np.abs(Ll) @ np.abs(Ll.T)))


@pytest.mark.parametrize("bad", [0, 3, 7, 8, 15])
def test_failing_pivot(block16, bad):
    A = spd(16, 5)
    A[bad, bad] = -1.0
    L, M, info = block16(A, True)
    assert info == bad and L[bad, bad] == 1.0


@pytest.mark.parametrize("cols", [3, 8, 11, 16])
@pytest.mark.parametrize("down", [False, True])
def test_inverse_in_place(block16, cols, down):
    L = np.linalg.cholesky(spd(cols, 40 + cols))
    _, M, info = block16(L, False, cols, down)
    assert info == -1
    assert np.allclose(np.tril(M) @ L, np.eye(16), rtol=0, atol=1e-13)
    _, Mi, info = block16(L, False, cols, down, in_place=True)
    assert info == -1 and np.array_equal(np.tril(Mi), np.tril(M))


@pytest.mark.parametrize("seed", range(8))
def test_inverse_residual(block16, seed):
    # ill-conditioned 8 x 8 diagonal blocks (9e5), L21 = K2 Z K1
    rng = np.random.default_rng(seed)
    c, s = np.cos(0.3), np.sin(0.3)
    K1, K2 = ((np.eye(8) - c * np.tril(np.ones((8, 8)), -1)) * s ** np.arange(8) * (1 + 0.1 * rng.random((8, 8)))
              for _ in range(2))
    L = np.block([[K1, np.zeros((8, 8))], [K2 @ rng.standard_normal((8, 8)) @ K1, K2]])
    _, M, info = block16(L, False)
    assert info == -1
    L, M = L.astype(np.longdouble), np.tril(M).astype(np.longdouble)
    # column substitution: |L M - I| <= gamma_n |L| |M|, with a rounded
    # reciprocal and a product in place of a division
    assert np.all(np.abs(L @ M - np.eye(16)) <= 20 * U * (np.abs(L) @ np.abs(M)))

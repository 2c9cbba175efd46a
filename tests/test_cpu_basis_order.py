"""The elements of a Krylov basis vector that a product of the persistent
resistive solve reads from other threads: the same bits whichever of their
owners have stored theirs already (no barrier lies between the owners'
correction and the product), and the bits the owners store."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = os.path.join(str(tmp_path_factory.mktemp("basis")), "libbasis.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC",
                    os.path.join(ROOT, "tests", "basis_host.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("n,j", [(1, 0), (257, 1), (300, 2), (513, 29)])
def test_elements_do_not_depend_on_their_owners_progress(lib, n, j):
    rng = np.random.Generator(np.random.PCG64(n + j))
    w, V, d = rng.standard_normal(n), rng.standard_normal((j + 1, n)), 1e-3 * rng.standard_normal(j + 1)
    div = 0.7
    idx = rng.integers(0, n, 4 * n)
    reads = []
    for share in (0.0, 0.5, 1.0):
        gone = np.flatnonzero(rng.random(n) < share)
        Vs, out = V.copy(), np.empty(idx.size)
        w_before = w.copy()
        lib.basis_read(C.c_int64(n), j, _p(w), C.c_double(div), _p(Vs), _p(d), _p(gone), C.c_int64(gone.size), _p(idx),
                       C.c_int64(idx.size), _p(out))
        assert np.array_equal(w, w_before)
        reads.append(out)
    assert np.array_equal(reads[0], reads[1]) and np.array_equal(reads[0], reads[2])
    assert np.array_equal(reads[2], Vs[j][idx])  # what the owners stored
    s = w.copy()
    for c in range(j):
        s -= d[c] * V[c]
    assert np.array_equal(reads[0], (s / div)[idx])

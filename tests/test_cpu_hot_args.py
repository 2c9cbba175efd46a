"""The hot kernels' point arithmetic on the host: multiply-shift quotients
against integer division over every divisor a block extent can be (and the
largest), at the numerators around every multiple and at the ends of the
31-bit range, and the plane table against the field table."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = os.path.join(str(tmp_path_factory.mktemp("hot")), "libhot.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-D__host__=", "-D__device__=", "-D__forceinline__=inline",
                    os.path.join(ROOT, "tests", "hot_host.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def test_quotients(lib):
    ends = np.array([0, 1, 2, 2**31 - 2, 2**31 - 1], dtype=np.uint64)
    rng = np.random.Generator(np.random.PCG64(3))
    for d in list(range(1, 2100)) + [4095, 4096, 4097, 65535, 65536, 65537, 2**30 - 1, 2**30, 2**31 - 1]:
        m = np.unique(rng.integers(0, (2**31 - 1) // d + 1, 200, dtype=np.uint64)) * d
        t = np.unique(np.concatenate([ends, m, m + d - 1, np.where(m > 0, m - 1, 0)]))
        t = t[t < 2**31].astype(np.uint32)
        q = np.empty_like(t)
        lib.hot_quot(C.c_uint32(d), t.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p), len(t))
        assert np.array_equal(q, t // np.uint32(d)), d


def test_planes(lib):
    from beta1_b200 import mhd
    q = 0
    for f, (_, _, ncomp, _) in enumerate(mhd.field_table()):
        assert lib.hot_plane_of(f) == q
        q += ncomp


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 5), (1, 33, 4), (8, 6, 31), (5, 1, 32)])
@pytest.mark.parametrize("G", [4, 5])
def test_weight_order(lib, n, G):
    """every padded point has one place, the inner cells come first in their
    own order, the place leads back to the point, and no two values of a
    field share an index below the size of its planes"""
    ext = [x + 1 + 2 * G for x in n]
    vol = int(np.prod(ext))
    cell, back = np.empty(vol, np.int64), np.empty(vol, np.int64)
    lib.weight_order(*n, G, cell.ctypes.data_as(C.c_void_p), back.ctypes.data_as(C.c_void_p))
    assert np.array_equal(np.sort(cell), np.arange(vol))
    assert np.array_equal(back, np.arange(vol))
    inner = cell.reshape(ext)[G:G + n[0], G:G + n[1], G:G + n[2]]
    assert np.array_equal(inner.ravel(), np.arange(inner.size))
    lib.weight_value.restype = C.c_int64
    for nc in (18, 36):
        at = {lib.weight_value(C.c_int64(int(d)), nc, m) for d in (0, 31, 32, vol - 1) for m in range(nc)}
        assert len(at) == nc * len({0, 31, 32, vol - 1})
        assert max(at) < nc * (-(-vol // 32) * 32)

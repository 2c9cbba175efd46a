"""An upload may return without a wait only where the copy has read its source
by then: pageable memory, on a system whose device does not read pageable
memory itself (there the runtime need not stage the copy)."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = os.path.join(str(tmp_path_factory.mktemp("upload")), "libupload.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(ROOT, "tests", "upload_host.cpp"), "-o",
                    out], check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("unregistered,reads_pageable,early", [(1, 0, 1), (1, 1, 0), (0, 0, 0), (0, 1, 0)])
def test_rule(lib, unregistered, reads_pageable, early):
    assert lib.upload_rule(unregistered, reads_pageable) == early

"""The linear solver's walk over a matrix row (csrc/csr_rows.hpp) visits each
entry once, also at the end of the largest matrix that the library takes, whose
positions reach 2^31 - 2.  CPU only."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, REPO


@pytest.mark.parametrize("length", [0, 1, 9, 35, 36, 37, 95])
@pytest.mark.parametrize("end", [1000, 2 ** 31 - 2])
def test_each_entry_once(tmp_path, length, end):
    out = tmp_path / "librows.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(PKG_DIR, "csrc"), "-o", str(out),
                    os.path.join(REPO, "tests", "csr_rows_host.cpp")], check=True)
    walk = C.CDLL(str(out)).walk
    walk.restype, walk.argtypes = C.c_long, [C.c_int, C.c_int, C.c_void_p]
    seen = np.zeros(length + 1, np.uint8)
    assert walk(end - length, end, seen.ctypes.data) <= 4 * (length // 36 + 1)
    assert (seen[:length] == 1).all() and seen[length] == 0

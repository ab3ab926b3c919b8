"""Work on a second stream is joined to the first one on every way out of the
call that started it (csrc/stream_fork.hpp), over fakes of the CUDA calls.  CPU
only."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import PKG_DIR, REPO

FORK = "record f on m;s waits f;"
JOIN = "record j on s;m waits j;"


@pytest.fixture(scope="module")
def log(tmp_path_factory):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    out = tmp_path_factory.mktemp("fork") / "libfork.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",  # the fakes, not a loaded CUDA runtime
                    "-I" + os.path.join(PKG_DIR, "csrc"),
                    "-I" + os.path.join(cuda, "include"), "-o", str(out),
                    os.path.join(REPO, "tests", "stream_fork_host.cpp")], check=True)
    f = C.CDLL(str(out)).stream_fork_log
    f.restype, f.argtypes = C.c_char_p, [C.c_char_p, C.c_int]
    return lambda fail, work: f(fail.encode(), work).decode()


@pytest.mark.parametrize("fail,work,want", [
    ("", 0, FORK + "work;" + JOIN),
    # the call fails between the fork and the join: still joined, once
    ("", 1, FORK + "work;" + JOIN + "error;"),
    # the join itself fails: the host waits for the second stream
    ("record j on s", 0, FORK + "work;record j on s;synchronize s;error;"),
    ("m waits j", 0, FORK + "work;" + JOIN + "synchronize s;error;"),
    ("m waits j", 1, FORK + "work;" + JOIN + "synchronize s;error;"),
    # no fork, nothing to join
    ("s waits f", 0, FORK + "error;"),
])
def test_joined_on_every_way_out(log, fail, work, want):
    assert log(fail, work) == want

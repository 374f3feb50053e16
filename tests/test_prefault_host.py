"""The touch of output pages ahead of a copy (csrc/rq_prefault.h): every page becomes
resident, and no byte changes (a call that fails later leaves its caller's arrays alone)."""
import ctypes as C
import mmap
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "bayesian-rans-uq_b200" / "csrc"
SOURCE = """
#include "rq_prefault.h"
#include <cstdint>
#include <sys/mman.h>
#include <unistd.h>
#include <vector>
extern "C" void touch(void *p, size_t n) { rqc::prefault(p, n); }
extern "C" long missing(void *p, size_t n) {
    const uintptr_t size = sysconf(_SC_PAGESIZE), a = reinterpret_cast<uintptr_t>(p) / size * size;
    const size_t pages = (reinterpret_cast<uintptr_t>(p) + n - a + size - 1) / size;
    std::vector<unsigned char> in(pages);
    if (mincore(reinterpret_cast<void *>(a), pages * size, in.data()))
        return -1;
    long k = 0;
    for (unsigned char v : in)
        k += !(v & 1);
    return k;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("prefault")
    (d / "p.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC), "-o",
                    str(d / "p.so"), str(d / "p.cpp")], check=True)
    lib = C.CDLL(str(d / "p.so"))
    lib.missing.restype = C.c_long
    return lib


@pytest.mark.parametrize("offset,size", [(0, 1), (0, 4096), (4095, 2), (8, 100000), (1000, 4096)])
def test_pages_are_touched_and_bytes_kept(lib, offset, size):
    m = mmap.mmap(-1, 40 * 4096)
    buf = np.frombuffer(m, dtype=np.uint8)
    p, n = C.c_void_p(buf.ctypes.data + offset), C.c_size_t(size)
    lib.touch(p, n)
    assert lib.missing(p, n) == 0
    buf[:] = np.random.default_rng(size).integers(0, 256, buf.size, dtype=np.uint8)
    want = buf.copy()
    lib.touch(p, n)
    np.testing.assert_array_equal(buf, want)


def test_nothing_to_touch(lib):
    lib.touch(None, C.c_size_t(0))

"""rr_host_gather without the memory for a thread (CPU): the calling thread
copies that part itself, and no exception leaves the C entry.  Built here from
the library's source with an allocator that refuses, in a process of its own."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SHIM = r"""
#include <cstdlib>
#include <new>
#include "%s/redrock_b200/csrc/rr_host.cpp"
extern "C" int allowed = 1 << 30;   // allocations until operator new refuses
void* operator new(std::size_t n) {
  if (allowed-- <= 0) throw std::bad_alloc();
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
"""
RUN = """
import ctypes, sys
import numpy as np
lib = ctypes.CDLL(sys.argv[1])
a = np.random.default_rng(0).integers(0, 255, 40 << 20, dtype=np.uint8)
for allowed in (0, 1, 3):
    out = np.zeros_like(a)
    src = np.array([a.ctypes.data], dtype=np.uintp)
    size = np.array([a.nbytes], dtype=np.int64)
    ctypes.c_int.in_dll(lib, "allowed").value = allowed
    rc = lib.rr_host_gather(ctypes.c_void_p(src.ctypes.data), ctypes.c_void_p(size.ctypes.data),
                            ctypes.c_int64(1), ctypes.c_void_p(out.ctypes.data),
                            ctypes.c_int64(out.nbytes))
    assert rc == 0 and np.array_equal(out, a), allowed
print("ok")
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_no_memory_for_threads(tmp_path):
    src, so = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text(SHIM % ROOT)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic",
                    "-o", str(so), str(src)], check=True)
    r = subprocess.run([sys.executable, "-c", RUN, str(so)], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]

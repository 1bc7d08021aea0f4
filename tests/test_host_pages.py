"""Result buffers: pages are populated once, and only looked up when present.

csrc/mnad_pages.h is compiled with the host compiler, its madvise counted."""
import ctypes as C
import mmap
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mnad-modeling-rtm_gb300", "csrc")

SHIM = r"""
#include <sys/mman.h>
#include <cstring>
static int calls = 0;
static int counted(void* p, size_t n, int what) { ++calls; return madvise(p, n, what); }
#define madvise counted
#include "mnad_pages.h"
#undef madvise
extern "C" int populate(char* p, size_t n) { calls = 0; mnad::populate_pages(p, n); return calls; }
extern "C" long present(char* p, size_t pages, size_t page)
{
    std::vector<unsigned char> v(pages);
    if (mincore(p, pages * page, v.data())) return -1;
    long k = 0;
    for (unsigned char x : v) k += x & 1;
    return k;
}
extern "C" char* map(size_t n)
{
    char* p = (char*)mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    return p;
}
extern "C" void unmap(char* p, size_t n) { munmap(p, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not hasattr(mmap, "MADV_DONTNEED"):
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("pages")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    L.map.restype = C.c_void_p
    L.present.restype = C.c_long
    for f in (L.populate, L.unmap):
        f.argtypes = [C.c_void_p, C.c_size_t]
    L.present.argtypes = [C.c_void_p, C.c_size_t, C.c_size_t]
    L.map.argtypes = [C.c_size_t]
    return L


@pytest.mark.parametrize("mb,off,cut", [(1, 0, 0), (4, 24, 8), (8, 4096 + 8, 1000), (29, 0, 16)])
def test_populated_once(lib, mb, off, cut):
    page, n = mmap.PAGESIZE, mb << 20
    p = lib.map(n)
    C.memset(p + off, 7, 1)                     # one page is present, the rest is fresh
    first = lib.populate(p + off, n - off - cut)
    if lib.present(p, n // page, page) < n // page - 2:
        lib.unmap(p, n)
        pytest.skip("the kernel has no MADV_POPULATE_WRITE")
    assert first == 1
    assert C.string_at(p + off, 1) == b"\x07" and C.string_at(p + off + 1, 64) == bytes(64)
    C.memset(p, 9, n)
    assert lib.populate(p + off, n - off - cut) == 0          # the second download
    assert C.string_at(p, n) == b"\x09" * n
    lib.unmap(p, n)
    lib.populate(p, n)                          # no longer mapped: nothing happens


@pytest.mark.parametrize("n", [0, 1000, (256 << 10) - 1, (30 << 20) + 1])
def test_sizes_left_to_the_copy(lib, n):
    p = lib.map(32 << 20)
    assert lib.populate(p, n) == 0 and lib.populate(None, 1 << 20) == 0
    lib.unmap(p, 32 << 20)

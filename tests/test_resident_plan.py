"""CPU checks of how the on-chip step kernel splits a grid over CTAs.

csrc/mnad_resident.h is compiled with the host compiler.  For grids from one
4-row group to the largest that fits, the patches must cover the grid exactly
once, fit an SM's shared memory, and every halo cell of a patch must find an
owner that publishes it, in a slot of its own; a patch that reads cells of
another must publish cells to it (the exchange's proof that no published word
is overwritten before it was read rests on that).
"""
import ctypes as C
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mnad-modeling-rtm_gb300", "csrc")

SHIM = r"""
#include "mnad_resident.h"
using namespace mnad;
extern "C" int plan(int nz, int nx, int d, int ncta, int* patches, int* bands, int* info)
{
    const ResPlan p = res_plan(nz, nx, d, ncta);
    for (size_t k = 0; k < p.patches.size(); ++k) {
        const ResPatch& q = p.patches[k];
        const int v[4] = {q.j0, q.nj, q.i0, q.ni};
        for (int m = 0; m < 4; ++m) patches[4 * k + m] = v[m];
    }
    for (size_t k = 0; k < p.band_first.size(); ++k) bands[k] = p.band_first[k];
    info[0] = (int)p.band_first.size() - 1; info[1] = (int)p.smem; info[2] = p.slots; info[3] = p.threads;
    return (int)p.patches.size();
}
extern "C" void layout(int j0, int nj, int i0, int ni, int nz, int nx, int d, int* o)
{
    const ResLayout L = res_layout(ResPatch{j0, nj, i0, ni}, nz, nx, d);
    const int v[18] = {L.fs, L.xleft, L.xcols, L.zt, L.zb, L.zb_first, L.nquads, L.nhalo, L.r, L.xm, L.ztm, L.zbm,
                       L.inj, L.qtab, L.qinj, L.halo, L.recs, L.total};
    for (int k = 0; k < 18; ++k) o[k] = v[k];
}
extern "C" int slot(int nj, int ni, int lr, int lc) { return res_slot(nj, ni, lr, lc); }
"""
NAMES = ("fs", "xleft", "xcols", "zt", "zb", "zb_first", "nquads", "nhalo", "r", "xm", "ztm", "zbm", "inj", "qtab",
         "qinj", "halo", "recs", "total")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("resident")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def get_plan(lib, nz, nx, d, ncta):
    pa, ba, info = (C.c_int * 4096)(), (C.c_int * 256)(), (C.c_int * 4)()
    n = lib.plan(nz, nx, d, ncta, pa, ba, info)
    return np.array(pa[:4 * n]).reshape(n, 4), list(ba[:info[0] + 1]), info[1], info[2], info[3]


def get_layout(lib, p, nz, nx, d):
    o = (C.c_int * 18)()
    lib.layout(*[int(x) for x in p], nz, nx, d, o)
    return dict(zip(NAMES, o))


def halo_cells(p, nz, nx):
    j0, nj, i0, ni = (int(x) for x in p)
    cells = [(j0 + r, i0 + c) for c in (-2, -1, ni, ni + 1) for r in range(nj)]
    cells += [(j0 + r, i0 + c) for r in (-2, -1, nj, nj + 1) for c in range(ni)]
    cells += [(j0 + r, i0 + c) for r in (-1, nj) for c in (-1, ni)]
    return [(j, i) for j, i in cells if 0 <= j < nz and 0 <= i < nx]


GRIDS = [(481, 1281, 40, 152), (381, 681, 40, 152), (201, 201, 20, 152), (96, 112, 10, 152), (4, 1, 0, 152), (5, 7, 1, 152),
         (64, 16, 6, 152), (150, 100, 12, 7), (256, 256, 20, 19), (1000, 33, 8, 152), (33, 2000, 8, 152), (129, 3, 1, 4),
         (80, 80, 40, 152), (127, 700, 0, 30), (260, 80, 30, 3)]


def random_grids():
    r = random.Random(1)
    out = []
    for _ in range(25):
        d = r.choice([0, 3, 10, 20, 40])
        out.append((2 * d + r.randint(1, 400), 2 * d + r.randint(1, 600), d, r.choice([1, 2, 5, 19, 76, 152])))
    return out


@pytest.mark.parametrize("nz,nx,d,ncta", GRIDS + random_grids())
def test_patches_cover_the_grid_and_exchange_their_edges(lib, nz, nx, d, ncta):
    patches, bands, smem, slots, threads = get_plan(lib, nz, nx, d, ncta)
    if len(patches) == 0:                       # only where the state is too large for so few CTAs
        assert nz * nx * 28 > 0.3 * ncta * 227 * 1024
        return
    assert len(patches) <= ncta and threads % 32 == 0 and 128 <= threads <= 512
    rows = (nz + 3) // 4 * 4
    owner = np.full((rows, nx), -1)
    for k, (j0, nj, i0, ni) in enumerate(patches):
        assert j0 % 4 == 0 and nj % 4 == 0 and 4 <= nj <= 128 and 1 <= ni <= 255
        assert (owner[j0:j0 + nj, i0:i0 + ni] == -1).all()
        owner[j0:j0 + nj, i0:i0 + ni] = k
        L = get_layout(lib, (j0, nj, i0, ni), nz, nx, d)
        assert 4 * L["total"] <= smem <= 227 * 1024 - 1024
        # strips: every point of the patch in a strip has its variables
        assert L["xcols"] == sum(1 for i in range(i0, i0 + ni) if i < d or i >= nx - d)
        assert L["xleft"] == sum(1 for i in range(i0, i0 + ni) if i < d)
        assert L["zt"] == 4 * sum(1 for j in range(j0, j0 + nj, 4) if j < d)
        assert L["zb"] == (4 * sum(1 for j in range(j0, j0 + nj, 4) if j + 3 >= nz - d) if d else 0)
        order = [L[n] for n in ("r", "xm", "ztm", "zbm", "inj", "qtab", "qinj", "halo", "recs", "total")]
        assert order == sorted(order) and L["r"] == 6 * L["fs"]
        assert L["halo"] % 4 == 0 and L["recs"] % 2 == 0 and L["inj"] % 4 == 0
    assert (owner >= 0).all()
    reads = set()
    for k, p in enumerate(patches):
        cells = halo_cells(p, nz, nx)
        assert len(cells) <= get_layout(lib, p, nz, nx, d)["nhalo"]
        seen = set()
        for j, i in cells:
            # the kernel's search: the band of the row, then the patch of the column
            b = max(b for b in range(len(bands) - 1) if patches[bands[b]][0] <= j)
            o = max(q for q in range(bands[b], bands[b + 1]) if patches[q][2] <= i)
            assert o == owner[j, i] != k
            j0, nj, i0, ni = (int(x) for x in patches[o])
            s = lib.slot(nj, ni, j - j0, i - i0)
            assert 0 <= s < slots and (o, s) not in seen
            seen.add((o, s))
            # ... which the owner's group at that cell writes
            lc, lr = i - i0, j - j0
            if lc < 2 or lc >= ni - 2:
                assert s == (lc if lc < 2 else lc - ni + 4) * nj + lr
            else:
                zq, row = lr // 4, lr % 4
                assert (zq == 0 and row < 2) or (zq == nj // 4 - 1 and row >= 2)
                assert s == 4 * nj + lc + (row if zq == 0 and row < 2 else row) * ni
            reads.add((k, int(o)))
    assert all((b, a) in reads for a, b in reads)


def test_no_two_cells_of_a_patch_share_a_slot(lib):
    for nj in (4, 8, 12, 128):
        for ni in (1, 2, 3, 4, 5, 40):
            s = [lib.slot(nj, ni, r, c) for r in range(nj) for c in range(ni)]
            s = [x for x in s if x >= 0]
            assert len(s) == len(set(s)) and max(s) < 4 * nj + 4 * ni


def test_a_grid_too_large_for_the_sms_has_no_plan(lib):
    assert len(get_plan(lib, 1281, 4081, 40, 152)[0]) == 0

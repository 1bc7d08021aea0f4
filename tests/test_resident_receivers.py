"""Receivers beyond a patch's own table make a step of the on-chip kernel look up
all of them; MNAD_KERNEL_AUTO takes the other kernel where that costs more.

CPU: the count of receivers per patch, against a count cell by cell; the
estimate, against measured times.  GPU: which kernel runs, and the same bits.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mnad-modeling-rtm_gb300", "csrc")
SMS = 152

SHIM = r"""
#include "mnad_resident.h"
using namespace mnad;
extern "C" int most(int nz, int nx, int d, int ncta, int nr, const int* zr, const int* xr, int* slow)
{
    const ResPlan p = res_plan(nz, nx, d, ncta);
    if (!p.ok()) return -1;
    const std::vector<int> z(zr, zr + nr), x(xr, xr + nr);
    int held = 0;
    for (const ResPatch& q : p.patches) {
        int n = 0;
        for (int k = 0; k < nr; ++k) n += z[k] >= q.j0 && z[k] < q.j0 + q.nj && x[k] >= q.i0 && x[k] < q.i0 + q.ni;
        held = std::max(held, n);
    }
    *slow = held;
    return res_most_receivers(p, z, x);
}
extern "C" int pays(int nz, int nx, int d, int n, int wave, int sms, int tile_cols, int steps, int nr, int forward)
{
    const ResPlan p = res_plan(nz, nx, d, sms / wave);
    return res_pays(p, wave, sms, nz, nx, d, tile_cols,
                    std::vector<ResRun>(n, ResRun{steps, 0, false, res_scan_us(nr, p.comm, forward != 0)}));
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("receivers")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", so], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("nz,nx,d,ncta", [(201, 201, 20, 152), (321, 641, 40, 76), (9, 7, 0, 152), (130, 700, 12, 60), (481, 1281, 40, 152)])
def test_receivers_per_patch(lib, nz, nx, d, ncta):
    rng = np.random.default_rng(nz)
    for nr in (0, 1, 700):
        zr = np.concatenate([rng.integers(0, nz, nr), [0, nz - 1, 0, nz - 1], np.full(nx, nz // 2)]).astype(np.int32)
        xr = np.concatenate([rng.integers(0, nx, nr), [0, nx - 1, nx - 1, 0], np.arange(nx)]).astype(np.int32)
        slow = C.c_int()
        p = lambda a: a.ctypes.data_as(C.POINTER(C.c_int))      # noqa: E731
        n = lib.most(nz, nx, d, ncta, zr.size, p(zr), p(xr), C.byref(slow))
        assert n == slow.value > 0


# receivers on a square block in the middle of the grid: (grid, propagations, per launch,
# tile columns, receivers, forward), us a step on chip and without
@pytest.mark.parametrize("nz,nx,d,n,wave,tile,nr,forward,chip,other", [
    (201, 201, 20, 1, 1, 0, 576, 1, 2.15, 4.49), (201, 201, 20, 1, 1, 0, 4096, 1, 12.9, 4.63),
    (201, 201, 20, 8, 8, 0, 400, 1, 7.04, 11.88), (201, 201, 20, 8, 8, 0, 1600, 1, 22.0, 12.1),
    (321, 641, 40, 1, 1, 0, 576, 1, 5.06, 8.15), (321, 641, 40, 1, 1, 0, 1600, 1, 10.2, 8.16),
    (481, 1281, 40, 1, 1, 0, 784, 1, 12.3, 16.6), (481, 1281, 40, 1, 1, 0, 1600, 1, 21.9, 16.6),
    (481, 1281, 40, 4, 1, 16, 784, 1, 50.3, 31.7), (321, 641, 40, 1, 1, 0, 4096, 0, 16.7, 9.0),
    (481, 1281, 40, 4, 1, 16, 1600, 0, 51.6, 37.7)])
def test_looking_them_up_is_weighed(lib, nz, nx, d, n, wave, tile, nr, forward, chip, other):
    assert lib.pays(nz, nx, d, n, wave, SMS, tile, 1000, nr, forward) == int(chip < other)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,points,kernel", [("model", 14, "resident"), ("model", 60, "direct"), ("rtm", 60, "direct")])
def test_which_kernel_runs(kind, points, kernel):
    import mnad
    from mnad import build, workflow
    build.build()
    nz, nx, d, nt = 201, 180, 20, 50
    v = np.asfortranarray(1800.0 + 500.0 * np.random.default_rng(1).random((nz, nx)))
    zr, xr = (a.ravel().astype(float) for a in np.mgrid[60:60 + points, 60:60 + points])
    out = {}
    for k in ("auto", "direct"):
        j = mnad.ShotJob(kind, v, 10.0, 10.0, 1e-3, nt, d, 80.0, 90.0, zr, xr, workflow.ricker(28.0, 1e-3, nt),
                         vs=0.97 * v if kind == "rtm" else None, T=5 if kind == "rtm" else 0)
        with mnad.Context(0, kernel=k) as ctx:
            p = ctx.plan([j])
            p.run()
            p.download()
            assert p.kernels()["forward"] == (kernel if k == "auto" else "direct")
            p.close()
        out[k] = [a for a in (j.data, j.image, j.illum) if a is not None]
    for a, b in zip(out["auto"], out["direct"]):
        assert np.abs(b).max() > 0
        assert np.array_equal(a, b)

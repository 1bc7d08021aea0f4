"""No split of a grid asks for more shared memory or threads than the on-chip
kernel's launch can have, whichever layout its patches take.

csrc/mnad_resident.h is compiled with the host compiler and swept over grids,
CPML widths and CTA counts: thin grids and patches of a few hundred points,
where the table with an entry per point is largest beside the state, are where
a split can outgrow an SM.  The GPU test runs such grids by default and
compares them with the kernel they would take without the on-chip one.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mnad-modeling-rtm_gb300", "csrc")
SMEM = 227 * 1024 - 1024              # a CTA's shared memory less the kernel's static part
SMS = 152

SHIM = r"""
#include "mnad_resident.h"
using namespace mnad;
// out: patches, largest shared memory of a patch in the layout the plan runs,
// smem and threads of the plan, 1 if it goes point by point, 1 if an area is misaligned
static void look(int nz, int nx, int d, int ncta, int* out)
{
    const ResPlan p = res_plan(nz, nx, d, ncta);
    size_t most = 0;
    int off = 0;
    for (const ResPatch& q : p.patches) {
        const ResLayout L = res_layout(q, nz, nx, d, p.small);
        most = std::max(most, (size_t)L.total * 4);
        for (int o : {L.fs, L.r, L.xm, L.ztm, L.zbm, L.xk, L.ztk, L.zbk, L.inj, L.qtab, L.halo}) off |= o % 4 != 0;
        off |= L.recs % 2 != 0;
    }
    const int v[6] = {(int)p.patches.size(), (int)most, (int)p.smem, p.threads, p.small, off};
    for (int k = 0; k < 6; ++k) out[k] = v[k];
}
extern "C" void plan(int nz, int nx, int d, int ncta, int* out) { look(nz, nx, d, ncta, out); }
// every plan of the grids nz0, nz0 + dz, .. < nz1 by nx0, nx0 + dx, .. < nx1 on
// sms / m CTAs, m = 1 .. 24: plans found; the first one beyond a limit in `bad`
extern "C" long sweep(int nz0, int nz1, int dz, int nx0, int nx1, int dx, int d, int sms, long limit, int* bad)
{
    long n = 0;
    bad[0] = 0;
    for (int nz = nz0; nz < nz1; nz += dz)
        for (int nx = nx0; nx < nx1; nx += dx)
            for (int m = 1; m <= 24; ++m) {
                int o[6];
                look(nz, nx, d, sms / m, o);
                if (o[0] == 0) break;                       // nor on fewer CTAs
                ++n;
                const int cap = o[4] ? RES_POINT_THREADS : RES_THREADS;
                if (bad[0] == 0 && (o[1] > limit || o[2] != o[1] || o[3] > cap || o[3] % 32 || o[0] > sms / m || o[5])) {
                    bad[0] = nz; bad[1] = nx; bad[2] = sms / m;
                    for (int k = 0; k < 6; ++k) bad[3 + k] = o[k];
                }
            }
    return n;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("limits")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    L.sweep.restype = C.c_long
    return L


# (nz, nx, d, propagations of a launch): patches of up to 1024 points whose table
# with an entry per point does not fit beside the state
TIGHT = [(72, 205, 10, 6), (78, 161, 10, 8), (50, 269, 20, 4), (81, 629, 10, 2), (56, 1378, 8, 1), (4, 1159, 0, 8)]


@pytest.mark.parametrize("nz,nx,d,m", TIGHT)
def test_a_patch_whose_point_table_does_not_fit_goes_by_groups(lib, nz, nx, d, m):
    o = (C.c_int * 6)()
    lib.plan(nz, nx, d, SMS // m, o)
    patches, most, smem, threads, small, off = o
    assert patches > 0 and most == smem <= SMEM and threads <= 384 and not small and not off


@pytest.mark.parametrize("d", [0, 4, 10, 20, 40])
@pytest.mark.parametrize("nz,nx", [((4, 160, 7), (4, 400, 13)), ((4, 90, 5), (400, 3000, 131)), ((160, 700, 53), (20, 900, 97))])
def test_no_plan_is_beyond_the_limits(lib, nz, nx, d):
    bad = (C.c_int * 9)()
    lo = lambda r: max(r[0], 2 * d + 1)         # noqa: E731
    n = lib.sweep(lo(nz), nz[1], nz[2], lo(nx), nx[1], nx[2], d, SMS, C.c_long(SMEM), bad)
    assert n > 0
    assert bad[0] == 0, dict(zip(("nz", "nx", "ncta", "patches", "most", "smem", "threads", "small", "off"), bad))


@pytest.mark.gpu
@pytest.mark.parametrize("nz,nx,d,n", [(72, 205, 10, 6), (78, 161, 10, 8), (50, 269, 20, 4), (56, 1378, 8, 1)])
def test_such_grids_run_and_equal_the_other_kernel(nz, nx, d, n):
    import mnad
    from mnad import build, workflow
    build.build()
    rng = np.random.default_rng(nz)
    v = np.asfortranarray(1800.0 + 500.0 * rng.random((nz, nx)))
    xr = np.arange(1, nx + 1, dtype=float)
    out = {}
    # fewer than 2.25 tiles of 64 x 16 points per CTA: without the on-chip kernel, one thread per point
    assert n * ((nz + 63) // 64) * ((nx + 15) // 16) < 2.25 * 2 * SMS
    for kernel in ("auto", "direct"):
        jobs = [mnad.ShotJob("model", v, 10.0, 10.0, 1e-3, 60, d, float(d + 2), float(nx // 2 + k), np.full(nx, d + 2.0), xr,
                             workflow.ricker(28.0, 1e-3, 60)) for k in range(n)]
        with mnad.Context(0, kernel=kernel) as ctx:
            p = ctx.plan(jobs)
            p.run()
            p.download()
            assert p.kernels()["forward"] == ("resident" if kernel == "auto" else "direct")
            p.close()
        out[kernel] = [j.data for j in jobs]
    for a, b in zip(out["auto"], out["direct"]):
        assert np.linalg.norm(b) > 0
        assert np.array_equal(a, b)

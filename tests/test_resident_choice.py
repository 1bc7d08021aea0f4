"""When MNAD_KERNEL_AUTO takes the on-chip kernel for a group that would fit it.

csrc/mnad_resident.h estimates both sides (res_pays).  The CPU test holds the
rule against measured times on a GB300 of the on-chip kernel and of the kernel
that launches once per step: where one of them won by more than the estimates'
own error, the rule must pick it.  The GPU test runs groups on both sides of the
line and reads back which kernel ran; the outputs are the same bits either way.
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
// n propagations of `steps` steps, every second one with `snaps` snapshots; 2: no plan
extern "C" int pays(int nz, int nx, int d, int n, int wave, int sms, int tile_cols, int steps, int snaps, int f16)
{
    const ResPlan p = res_plan(nz, nx, d, sms / wave);
    if (!p.ok()) return 2;
    std::vector<ResRun> runs;
    for (int k = 0; k < n; ++k) runs.push_back(ResRun{steps, k % 2 ? snaps : 0, f16 != 0, 0.0});
    return res_pays(p, wave, sms, nz, nx, d, tile_cols, runs);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("choice")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", so], check=True)
    return C.CDLL(so)


# nz, nx, d, propagations, per launch, tile columns (0: one thread per point), steps, time on chip (us), time without
MEASURED = [
    # few steps between two returns to the host
    (64, 64, 20, 64, 50, 0, 4, 116, 63), (64, 64, 20, 64, 50, 0, 36, 365, 448),
    (201, 201, 20, 64, 10, 16, 4, 421, 234), (201, 201, 20, 64, 10, 16, 100, 3408, 5031),
    (321, 641, 40, 16, 2, 16, 6, 543, 347), (321, 641, 40, 16, 2, 16, 100, 3650, 5250),
    (128, 128, 20, 256, 25, 16, 12, 1271, 977), (128, 128, 20, 256, 25, 16, 100, 6593, 7794),
    (600, 1100, 20, 16, 1, 8, 12, 1664, 1207), (600, 1100, 20, 4, 1, 8, 6, 278, 200),
    (481, 1281, 40, 4, 1, 16, 6, 307, 223), (481, 1281, 40, 4, 1, 16, 100, 2021, 3250),
    (481, 1281, 40, 1, 1, 0, 240, 1260, 4040),
    # many steps: full SMs per propagation, strips in every patch, no strips at all
    (481, 1281, 40, 19, 1, 16, 1000, 92000, 128600), (481, 1281, 20, 10, 1, 8, 1000, 49400, 62700),
    (2000, 100, 0, 60, 3, 8, 104, 10347, 8604), (2000, 100, 40, 60, 1, 16, 104, 23935, 19994),
    (401, 901, 0, 33, 1, 8, 104, 11548, 9577), (780, 800, 0, 19, 1, 8, 104, 9909, 8724),
    (256, 256, 40, 46, 6, 16, 1000, 39300, 50000), (100, 400, 20, 75, 10, 16, 104, 4600, 6500),
    (33, 2000, 0, 91, 4, 8, 1000, 63500, 111300), (12, 5000, 2, 16, 1, 16, 200, 6675, 18770),
    (16, 16, 2, 1024, 152, 16, 100, 1131, 2817), (201, 201, 20, 4, 4, 0, 200, 650, 1584),
]


@pytest.mark.parametrize("nz,nx,d,n,wave,tile,steps,chip,other", MEASURED)
def test_the_faster_kernel_is_taken(lib, nz, nx, d, n, wave, tile, steps, chip, other):
    assert chip > 1.1 * other or other > 1.1 * chip
    assert lib.pays(nz, nx, d, n, wave, SMS, tile, steps, 0, 0) == int(chip < other)


# 32 forwards of 16 shots (true and background model by turns), 96 steps: time of a step of all (us)
@pytest.mark.parametrize("nz,nx,d,wave,tile,snaps,f16,chip,other", [
    (600, 1100, 20, 1, 8, 96, 1, 376.9, 322.4), (321, 641, 40, 2, 16, 96, 1, 212.1, 173.1),
    (481, 1281, 40, 1, 16, 96, 1, 367.9, 330.9), (481, 1281, 40, 1, 16, 24, 1, 216.3, 240.3),
    (481, 1281, 40, 1, 16, 12, 0, 175.0, 212.0), (201, 201, 20, 10, 16, 96, 1, 38.7, 88.8)])
def test_snapshots_are_weighed(lib, nz, nx, d, wave, tile, snaps, f16, chip, other):
    assert chip > 1.1 * other or other > 1.1 * chip
    assert lib.pays(nz, nx, d, 32, wave, SMS, tile, 96, snaps, f16) == int(chip < other)


@pytest.mark.gpu
@pytest.mark.parametrize("nz,nx,d,n,nt,kernel", [(201, 201, 20, 64, 6, "tma"), (201, 201, 20, 64, 60, "resident"),
                                                 (2000, 100, 40, 40, 30, "tma"), (600, 1100, 20, 8, 12, "tma_narrow")])
def test_which_kernel_runs(nz, nx, d, n, nt, kernel):
    import mnad
    from mnad import build, workflow
    build.build()
    v = np.asfortranarray(1800.0 + 500.0 * np.random.default_rng(nz).random((nz, nx)))
    xr = np.arange(1, nx + 1, 3, dtype=float)
    other = "tma_narrow" if kernel == "tma_narrow" else "tma"
    out = {}
    for k in ("auto", other):
        jobs = [mnad.ShotJob("model", v, 10.0, 10.0, 1e-3, nt, d, float(d + 2), float(1 + (7 * m) % nx), np.full(xr.size, d + 2.0),
                             xr, workflow.ricker(28.0, 1e-3, nt)) for m in range(n)]
        with mnad.Context(0, kernel=k) as ctx:
            p = ctx.plan(jobs)
            p.run()
            p.download()
            assert p.kernels()["forward"] == (kernel if k == "auto" else other)
            p.close()
        out[k] = [j.data for j in jobs]
    assert max(np.abs(a).max() for a in out[other]) > 0
    for a, b in zip(out["auto"], out[other]):
        assert np.array_equal(a, b)

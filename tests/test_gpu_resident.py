"""The on-chip step kernel (MNAD_KERNEL_RESIDENT, what MNAD_KERNEL_AUTO takes
where a propagation's state fits the SMs): bit for bit the outputs of the
kernel that AUTO would take without it -- one thread per point below 2.25
64 x 16 tiles per resident CTA, the persistent kernel from there on -- for
every event of the time loop, at patch edges, in one patch and in many.
"""
import numpy as np
import pytest

import mnad
from mnad import workflow
from oracle import coracle

pytestmark = pytest.mark.gpu
TOL_GATHER = 1e-5


@pytest.fixture(scope="module", autouse=True)
def built():
    from mnad import build
    build.build()


def rel(a, b):
    a, b = np.ravel(np.asarray(a), order="F"), np.ravel(np.asarray(b), order="F")
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def shot(nz, nx, d, nt, zs=None, xs=None, receivers="line", seed=0):
    rng = np.random.default_rng(seed)
    z = np.arange(nz)[:, None]
    v = np.where(z < nz // 2, 1700.0, 2400.0) + 150.0 * rng.random((nz, nx))
    if receivers == "line":
        xr = np.arange(1, nx + 1, dtype=float)
        zr = np.full(nx, float(min(nz, d + 2)))
    elif receivers == "field":                  # every point of a block: more than a patch's own table
        m = min(nz, 24), min(nx, 24)
        zr, xr = (a.ravel().astype(float) for a in np.mgrid[1:m[0] + 1, 1:m[1] + 1])
    else:                                       # depths and duplicates: several receivers at one point
        xr = np.array([1, 2, nx, nx - 1, nx // 2, nx // 2, nx // 2, nx // 3, nx // 3], dtype=float)
        zr = np.array([1, nz, 1, nz - 1, nz // 2, nz // 2, nz // 2 + 1, nz // 3, nz // 4 + 1], dtype=float)
        zr, xr = np.maximum(zr, 1), np.maximum(xr, 1)
    return dict(v=np.asfortranarray(v), vs=np.asfortranarray(0.97 * v + 40.0), dx=10.0, dz=10.0, dt=1e-3, nt=nt, d=d,
                zs=float(zs or min(nz, d + 2)), xs=float(xs or max(1, nx // 3)), xr=xr, zr=zr,
                w=workflow.ricker(28.0, 1e-3, nt))


def tiles(s, n=1):
    nz, nx = s["v"].shape
    return n * ((nz + 63) // 64) * ((nx + 15) // 16)


def other_kernel(s, n=1):
    return "tma" if tiles(s, n) >= 2.25 * 304 else "direct"


def plan(kernel, shots, kind, T=3, codec="f32", pairing="reference"):
    jobs = [mnad.ShotJob(kind, s["v"], s["dx"], s["dz"], s["dt"], s["nt"], s["d"], s["zs"], s["xs"], s["zr"], s["xr"],
                         s["w"], vs=s["vs"] if kind == "rtm" else None, T=T if kind == "rtm" else 0) for s in shots]
    with mnad.Context(0, kernel=kernel, snapshot_codec=codec, pairing=pairing) as ctx:
        p = ctx.plan(jobs)
        p.run()
        p.run()                                 # a second run starts from zero state again
        p.download()
        names = p.kernels()
        p.close()
    return [a for j in jobs for a in ((j.data, j.image, j.illum) if kind == "rtm" else (j.data,))], names


def same(shots, kind, **k):
    a, names = plan("auto", shots, kind, **k)
    assert names["forward"] == "resident"
    b, _ = plan(other_kernel(shots[0], len(shots) * (2 if kind == "rtm" else 1)), shots, kind, **k)
    for x, y in zip(a, b):
        assert np.all(np.isfinite(y))
        assert np.array_equal(x, y), rel(x, y)
    return a


# one patch, patches of a few columns, several bands, rows off the 4-row groups,
# strips as wide as the grid, patches large enough for inner columns, both roundings
@pytest.mark.parametrize("nz,nx,d,nt", [(9, 7, 0, 12), (8, 8, 2, 40), (33, 21, 4, 90), (70, 3, 1, 60), (5, 200, 2, 60),
                                        (130, 97, 12, 150), (129, 300, 40, 120), (402, 90, 30, 120),
                                        (200, 640, 20, 100), (481, 700, 40, 60), (590, 1195, 20, 40)])
def test_forward_equals_the_other_kernel(nz, nx, d, nt):
    out = same([shot(nz, nx, d, nt)], "model")
    assert np.linalg.norm(out[0]) > 0


@pytest.mark.parametrize("zs,xs", [(1, 1), (130, 97), (13, 12), (66, 49), (64, 16), (3, 90)])
def test_source_anywhere(zs, xs):
    same([shot(130, 97, 12, 120, zs=zs, xs=xs)], "model")


@pytest.mark.parametrize("receivers", ["line", "field", "deep"])
@pytest.mark.parametrize("codec,T", [("f32", 1), ("bf16", 3), ("f16", 1), ("f16", 4)])
def test_rtm_equals_the_other_kernel(receivers, codec, T):
    out = same([shot(150, 110, 12, 130, receivers=receivers)], "rtm", T=T, codec=codec)
    assert np.linalg.norm(out[1]) > 0


def test_rtm_of_large_patches_and_of_the_persistent_rounding():
    same([shot(250, 500, 20, 90, zs=130, xs=250)], "rtm", T=2)
    same([shot(250, 500, 20, 91, seed=k) for k in range(2)], "rtm", T=7, codec="f16")
    same([shot(420, 820, 20, 60, zs=200, xs=410, seed=k) for k in range(2)], "rtm", T=5, codec="bf16")


@pytest.mark.parametrize("receivers", ["field", "deep"])
def test_receivers_of_large_patches(receivers):
    """More receivers in a patch than its own table holds; several at one point."""
    same([shot(250, 500, 20, 70, receivers=receivers, zs=12, xs=14)], "rtm", T=3, codec="bf16")


@pytest.mark.parametrize("nt", [1, 2, 3])
def test_shortest_records(nt):
    same([shot(90, 60, 8, nt)], "rtm", T=1)


def test_batches_share_launches():
    """More propagations than one launch holds, record lengths of their own."""
    same([shot(64, 64, 6, 60 + 7 * k, seed=k, xs=8 + 5 * k) for k in range(7)], "model")
    same([shot(260, 520, 20, 50 + k, seed=k) for k in range(9)], "model")


# byte counts off 16 and off the pieces that are zeroed at a time; every buffer
# a run adds to (records, images, illumination, FP16 maxima)
@pytest.mark.parametrize("kernel", ["auto", "direct", "tma"])
@pytest.mark.parametrize("nz,nx,d,nt,codec", [(41, 37, 4, 33, "f32"), (151, 111, 13, 51, "f16"), (300, 257, 20, 40, "bf16")])
def test_a_run_leaves_nothing_to_the_next(kernel, nz, nx, d, nt, codec):
    s = shot(nz, nx, d, nt)
    out = []
    for runs in (1, 3):
        j = mnad.ShotJob("rtm", s["v"], s["dx"], s["dz"], s["dt"], s["nt"], s["d"], s["zs"], s["xs"], s["zr"], s["xr"],
                         s["w"], vs=s["vs"], T=2)
        with mnad.Context(0, kernel=kernel, snapshot_codec=codec) as ctx:
            p = ctx.plan([j])
            for _ in range(runs):
                p.run()
            p.download()
            p.close()
        out.append([j.data, j.image, j.illum])
    assert np.abs(out[0][1]).max() > 0
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_a_plan_of_resident_and_other_groups():
    """Both in one captured run; launches counted as issued."""
    shots = [shot(90, 90, 8, 40), shot(1000, 1300, 8, 40)]
    out = {}
    for kernel in ("auto", "direct"):
        jobs = [mnad.ShotJob("model", s["v"], s["dx"], s["dz"], s["dt"], s["nt"], s["d"], s["zs"], s["xs"], s["zr"],
                             s["xr"], s["w"]) for s in shots]
        with mnad.Context(0, kernel=kernel) as ctx:
            p = ctx.plan(jobs)
            p.run()
            p.run()
            p.download()
            assert p.timing()["step_launches"] == 80
            assert p.launches() == (41 if kernel == "auto" else 80)
            p.close()
        out[kernel] = [j.data for j in jobs]
    assert np.array_equal(out["auto"][0], out["direct"][0])
    assert rel(out["auto"][1], out["direct"][1]) <= TOL_GATHER


def test_energy_fields_and_split_runs():
    """Host work between steps cuts a run into several launches."""
    s = shot(120, 140, 12, 101)
    a = (s["dx"], s["xs"], s["xr"], s["dz"], s["zs"], s["zr"], s["v"], s["dt"], s["nt"], s["w"], s["d"])
    got = {}
    for kernel in ("auto", "direct"):
        with mnad.Context(0, kernel=kernel, energy_every=7) as ctx:
            data, fields = ctx.fwd_fields(*a, [1, 2, 50, 101])
            got[kernel] = [data, ctx.energy()] + [f for t in sorted(fields) for f in fields[t]]
            got[kernel] += list(ctx.fwd(*a, record_vw=True)) + [ctx.energy()]
    for k, (x, y) in enumerate(zip(got["auto"], got["direct"])):
        if x.ndim == 1:                         # energies: FP64 atomics in any order
            assert np.allclose(x, y, rtol=1e-12, atol=0)
        else:
            assert np.array_equal(x, y), k


def test_checkpointed_rtm_equals_the_other_kernel():
    """Step windows of their own per propagation (odd starts, empty rounds)."""
    shots = [shot(130, 110, 10, 121 + 14 * k, seed=k) for k in range(2)]
    out = {}
    for kernel in ("auto", "direct"):
        jobs = [mnad.ShotJob("rtm", s["v"], s["dx"], s["dz"], s["dt"], s["nt"], s["d"], s["zs"], s["xs"], s["zr"],
                             s["xr"], s["w"], vs=s["vs"], T=3) for s in shots]
        with mnad.Context(0, kernel=kernel, checkpoint_every=30) as ctx:
            ctx.run_jobs(jobs)
        out[kernel] = [a for j in jobs for a in (j.data, j.image, j.illum)]
    for x, y in zip(out["auto"], out["direct"]):
        assert np.array_equal(x, y)


def test_a_wait_that_runs_out_returns_timeout_and_the_context_recovers():
    s = shot(200, 300, 20, 200)
    a = (s["dx"], s["xs"], s["xr"], s["dz"], s["zs"], s["zr"], s["v"], s["dt"], s["nt"], s["w"], s["d"])
    with mnad.Context(0) as ctx:
        ctx.set_wait_limit(1)
        with pytest.raises(mnad.MnadError) as e:
            ctx.fwd(*a)
        assert e.value.code == mnad._lib.E_TIMEOUT
        ctx.set_wait_limit(0)
        got = ctx.fwd(*a)
    ref = coracle.fwd(s["dx"], int(s["xs"]), s["xr"], s["dz"], int(s["zs"]), s["zr"], s["v"], s["dt"], s["nt"], s["w"],
                      s["d"])["datau"]
    assert rel(got, ref) <= TOL_GATHER


def test_no_room_for_the_exchange_takes_the_other_kernel():
    """A context whose budget holds the propagation but not the published cells."""
    s = shot(300, 500, 20, 60)
    a = (s["dx"], s["xs"], s["xr"], s["dz"], s["zs"], s["zr"], s["v"], s["dt"], s["nt"], s["w"], s["d"])
    with mnad.Context(0) as ctx:
        ref = ctx.fwd(*a)
    with mnad.Context(0, kernel="direct") as ctx:
        j = mnad.ShotJob("model", s["v"], s["dx"], s["dz"], s["dt"], s["nt"], s["d"], s["zs"], s["xs"], s["zr"], s["xr"],
                         s["w"])
        p = ctx.plan([j])
        held = ctx.memory()
        p.close()
    with mnad.Context(0, hbm_budget=held + (300 * 500 * 8) + (64 << 10)) as ctx:
        got = ctx.fwd(*a)
    assert np.array_equal(got, ref)

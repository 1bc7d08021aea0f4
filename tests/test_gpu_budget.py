"""A budget that suffices for a call on the one-thread-per-point kernel suffices
for it by default: the on-chip kernel's buffers take only room that is free, and
give it back to whatever the call allocates after them (outputs of the adjoint,
the next plan, a second launch group).  Outputs are the same bits at any budget.
"""
import numpy as np
import pytest

import mnad
from mnad import workflow

pytestmark = pytest.mark.gpu
NZ, NX, D, NT = 300, 500, 20, 24


@pytest.fixture(scope="module", autouse=True)
def built():
    from mnad import build
    build.build()


def shot(nz=NZ, nx=NX):
    v = np.asfortranarray(1800.0 + 500.0 * np.random.default_rng(3).random((nz, nx)))
    return dict(v=v, xr=np.arange(1, nx + 1, 2, dtype=float), zr=np.full((nx + 1) // 2, D + 2.0), w=workflow.ricker(28.0, 1e-3, NT))


def job(kind, s, T=4):
    return mnad.ShotJob(kind, s["v"], 10.0, 10.0, 1e-3, NT, D, D + 2.0, s["v"].shape[1] // 2, s["zr"], s["xr"], s["w"],
                        vs=s["v"] if kind == "rtm" else None, T=T if kind == "rtm" else 0)


def outputs(jobs):
    return [a.copy() for j in jobs for a in (j.data, j.image, j.illum) if a is not None]


def forward(ctx):
    s = shot()
    return [ctx.fwd(10.0, 200.0, s["xr"], 10.0, D + 2.0, s["zr"], s["v"], 1e-3, NT, s["w"], D)]


def rtm_calls(ctx):
    s = shot()
    ctx.set_options(T=4)
    d = ctx.fwd(10.0, 200.0, s["xr"], 10.0, D + 2.0, s["zr"], s["v"], 1e-3, NT, s["w"], D, ss=1, indx=1)
    return [d, ctx.adj(10.0, 10.0, NT, 1e-3, s["v"], s["xr"], s["zr"], d, D, ss=1)]


def jobs(ctx):
    ctx.set_options(snapshot_codec="f16")
    js = [job("rtm", shot()), job("model", shot(120, 140))]
    ctx.run_jobs(js)
    return outputs(js)


def two_plans(ctx):
    a, b = [job("rtm", shot())], [job("rtm", shot(280, 420))]
    p = ctx.plan(a)
    p.run()
    p.download()
    out = outputs(a)
    q = ctx.plan(b)                             # takes the room that the first one's buffers held
    for x, js in ((q, b), (p, a)):
        x.run()
        x.download()
        out += [v.copy() for v in x.stack()] + outputs(js)
    q.close()
    p.close()
    assert all(np.array_equal(x, y) for x, y in zip(out[:3], out[-3:]))
    return out


def checkpointed(ctx):
    ctx.set_options(checkpoint_every=8)
    js = [job("rtm", shot())]
    p = ctx.plan(js)
    p.run()
    p.run()
    p.download()
    p.close()
    return outputs(js)


def least_budget(kernel, call):
    """Smallest budget (16 KB steps) that the call runs in."""
    def runs(b):
        try:
            with mnad.Context(0, hbm_budget=b << 14, kernel=kernel) as ctx:
                return call(ctx)
        except mnad.MnadError as e:
            assert e.code == mnad._lib.E_BUDGET
            return None
    lo, hi = 1, 1 << 14
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if runs(mid) is not None else (mid, hi)
    return hi << 14, runs(hi)


@pytest.mark.parametrize("call", [forward, rtm_calls, jobs, two_plans, checkpointed])
def test_what_fitted_fits(call):
    need, ref = least_budget("direct", call)
    assert max(np.nanmax(np.abs(a)) for a in ref) > 0
    for more in [0, 16, 64, 160, 320, 512, 800, 1100, 1500, 2000, 3000, 4000, 6000, 8000, 12000]:
        with mnad.Context(0, hbm_budget=need + (more << 10)) as ctx:
            got = call(ctx)
            if call is not rtm_calls:           # (that one leaves its wavefield stored)
                assert np.array_equal(got[0], call(ctx)[0])
        for a, b in zip(got, ref):
            assert np.array_equal(a, b, equal_nan=True), more   # (a stack divides by the illumination, zero before any arrival)


def test_a_server_admits_what_it_admitted():
    def served(budget, kernel):
        js = [job("rtm", shot()), job("model", shot(120, 140)), job("rtm", shot())]
        with mnad.Server(0, hbm_budget_bytes=budget, chunk_steps=12, kernel=kernel) as srv:
            for t in [srv.submit(j) for j in js]:
                srv.wait(t, 60.0)
        return outputs(js)

    lo, hi, ref = 1, 1 << 10, None              # 256 KB steps
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            ref = served(mid << 18, "direct")
            hi = mid
        except mnad.MnadError as e:
            assert e.code == mnad._lib.E_BUDGET
            lo = mid
    for more in (0, 1, 2, 4, 8, 16, 40):
        for a, b in zip(served((hi + more) << 18, "auto"), ref):
            assert np.array_equal(a, b, equal_nan=True), more

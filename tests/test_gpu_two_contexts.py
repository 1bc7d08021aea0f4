"""Two contexts, and a server beside a context, on one GPU at once.

A launch of the on-chip kernel needs all the SMs it uses together, and its CTAs
wait for one another; the persistent kernel's launches overlap their
predecessors.  Run from several threads each call must give the bits it gives
alone, whatever the other stream runs: the on-chip kernel over all SMs, over a
few, or the persistent kernel.
"""
import threading

import numpy as np
import pytest

import mnad
from mnad import workflow

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from mnad import build
    build.build()


def shot(nz, nx, d, nt):
    v = np.asfortranarray(1800.0 + 500.0 * np.random.default_rng(nz).random((nz, nx)))
    xr = np.arange(1, nx + 1, 2, dtype=float)
    return (10.0, nx // 3, xr, 10.0, d + 2, np.full(xr.size, d + 3.0), v, 1e-3, nt, workflow.ricker(28.0, 1e-3, nt), d)


FULL, SMALL, PERSISTENT = shot(481, 1281, 40, 120), shot(150, 170, 20, 200), shot(1023, 1100, 20, 120)


def together(*work):
    errors = []

    def guarded(f):
        try:
            f()
        except Exception as e:                  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not any(t.is_alive() for t in threads)
    assert not errors, errors


@pytest.mark.parametrize("a,b", [(FULL, FULL), (FULL, SMALL), (PERSISTENT, FULL), (PERSISTENT, SMALL)])
def test_two_contexts(a, b):
    with mnad.Context(0) as A, mnad.Context(0) as B:
        alone = A.fwd(*a), B.fwd(*b)
        got = [], []
        together(lambda: got[0].extend(A.fwd(*a) for _ in range(6)), lambda: got[1].extend(B.fwd(*b) for _ in range(12)))
    for ref, outs in zip(alone, got):
        assert np.abs(ref).max() > 0 and len(outs) >= 6
        for o in outs:
            assert np.array_equal(o, ref)


def test_a_server_beside_a_context():
    def job(s):
        return mnad.ShotJob("model", s[6], s[0], s[3], s[7], s[8], s[10], s[4], s[1], s[5], s[2], s[9])
    with mnad.Context(0) as ctx, mnad.Server(0, hbm_budget_bytes=1 << 30, chunk_steps=32) as srv:
        ref = ctx.fwd(*FULL)
        served = srv.wait(srv.submit(job(SMALL)), 60.0).data.copy()
        outs, jobs = [], [job(SMALL) for _ in range(6)]
        together(lambda: outs.extend(ctx.fwd(*FULL) for _ in range(6)),
                 lambda: [srv.wait(t, 60.0) for t in [srv.submit(j) for j in jobs]])
    assert np.abs(served).max() > 0
    for o in outs:
        assert np.array_equal(o, ref)
    for j in jobs:
        assert np.array_equal(j.data, served)

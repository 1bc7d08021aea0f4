"""A server created with MNAD_KERNEL_TUNE runs the kernels of the automatic rule
(trial steps cannot run on live propagations): the on-chip kernel too, whose
exchange buffers show in the server's memory."""
import numpy as np
import pytest

import mnad
from mnad import workflow

pytestmark = pytest.mark.gpu


def test_tune_serves_as_auto():
    from mnad import build
    build.build()
    v = np.asfortranarray(1800.0 + 500.0 * np.random.default_rng(3).random((201, 201)))
    peak, out = {}, {}
    for kernel in ("auto", "tune", "direct"):
        j = mnad.ShotJob("model", v, 10.0, 10.0, 1e-3, 300, 20, 22.0, 90.0, np.full(160, 24.0), 21.0 + np.arange(160),
                         workflow.ricker(28.0, 1e-3, 300))
        with mnad.Server(0, hbm_budget_bytes=1 << 30, kernel=kernel) as srv:
            srv.wait(srv.submit(j), 60.0)
            peak[kernel] = srv.stats()["peak_bytes"]
        out[kernel] = j.data
    assert np.abs(out["auto"]).max() > 0
    assert np.array_equal(out["auto"], out["tune"]) and np.array_equal(out["auto"], out["direct"])
    assert peak["tune"] == peak["auto"] > peak["direct"]

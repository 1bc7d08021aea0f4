"""The table of what a batch zeroes at its start is built for batches that are
started as a whole only: not for the recomputed forwards of a checkpointed plan
(restored from checkpoints), and not for the server's batches (every propagation
starts by itself), whose tables would be built and uploaded at every admission.
"""
import numpy as np
import pytest

import mnad
from mnad import workflow

pytestmark = pytest.mark.gpu
PIECE = 64 << 10                                # bytes per 16-byte table entry


def uploaded(nr, nt):
    """Bytes copied to the device while a checkpointed plan of one RTM shot is created."""
    v = np.full((60, 70), 2000.0, order="F")
    j = mnad.ShotJob("rtm", v, 10.0, 10.0, 1e-3, nt, 8, 10.0, 30.0, np.full(nr, 12.0), 1.0 + np.arange(nr) % 70,
                     workflow.ricker(28.0, 1e-3, nt), vs=v, T=4)
    with mnad.Context(0, kernel="direct", checkpoint_every=16) as ctx:
        before = ctx.transfers()[0]
        p = ctx.plan([j])
        n = ctx.transfers()[0] - before
        p.close()
    return n


def test_no_table_for_the_recomputed_forwards():
    from mnad import build
    build.build()
    nr, a, b = 500, 400, 1200
    pieces = lambda nt, r: -(-nt * r * 8 // PIECE)              # noqa: E731
    # what grows with both the record and the receivers: the entries of the two forwards' records
    grown = (uploaded(nr, b) - uploaded(nr, a)) - (uploaded(1, b) - uploaded(1, a))
    assert grown == 2 * 16 * (pieces(b, nr) - pieces(a, nr) - (pieces(b, 1) - pieces(a, 1)))

"""A wait that runs out is named for what it may have waited for."""
import numpy as np
import pytest

import mnad
from mnad import workflow

pytestmark = pytest.mark.gpu


def test_the_message_names_the_on_chip_wait():
    from mnad import build
    build.build()
    v = np.full((200, 300), 2000.0, order="F")
    with mnad.Context(0) as ctx:
        ctx.set_wait_limit(1)
        with pytest.raises(mnad.MnadError) as e:
            ctx.fwd(10.0, 100, [50.0], 10.0, 30, [30.0], v, 1e-3, 60, workflow.ricker(28.0, 1e-3, 60), 20)
        assert e.value.code == mnad._lib.E_TIMEOUT
        assert "neighbour's cells" in str(e.value) and "tile copy" in str(e.value)

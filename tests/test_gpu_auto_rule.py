"""MNAD_KERNEL_AUTO where the on-chip kernel is not taken: the rule that chooses
between the kernels that launch once per step.  Groups that would fit are kept off
the chip by a block of 64 x 64 receivers, which it would look up at every step, the
large ones by their size; each runs the kernel the rule names, bit for bit."""
import numpy as np
import pytest

import mnad
from mnad import workflow

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from mnad import build
    build.build()


def jobs(nz, nx, d, n, nt):
    v = np.asfortranarray(1800.0 + 500.0 * np.random.default_rng(nz).random((nz, nx)))
    zr, xr = (a.ravel().astype(float) for a in np.mgrid[12:76, 12:76])
    return [mnad.ShotJob("model", v, 10.0, 10.0, 1e-3, nt, d, 40.0, float(20 + 11 * k % 60), zr, xr,
                         workflow.ricker(28.0, 1e-3, nt)) for k in range(n)]


def run(kernel, groups):
    js = [j for g in groups for j in jobs(*g)]
    with mnad.Context(0, kernel=kernel) as ctx:
        p = ctx.plan(js)
        p.run()
        p.download()
        names = p.kernels()["forward"]
        p.close()
    return [j.data for j in js], names


# 2.25 tiles of 64 x 16 points per resident CTA: 684 tiles; CPML strips under 15 % of the grid: narrow tiles
@pytest.mark.parametrize("group,kernel", [
    ((96, 112, 10, 3, 40), "direct"), ((700, 960, 12, 1, 20), "direct"),               # 42 and 660 tiles
    ((360, 376, 10, 5, 30), "tma_narrow"), ((201, 201, 30, 14, 30), "tma"),            # 720 and 728
    ((1000, 1300, 8, 1, 24), "tma_narrow"), ((1000, 1300, 60, 1, 24), "tma")])
def test_the_rule_without_the_on_chip_kernel(group, kernel):
    auto, name = run("auto", [group])
    assert name == kernel
    forced, same = run(kernel, [group])
    assert same == kernel
    for a, b in zip(auto, forced):
        assert np.abs(b).max() > 0
        assert np.array_equal(a, b)


def test_two_kernels_in_one_plan():
    small, large = (96, 112, 10, 3, 40), (1000, 1300, 8, 1, 40)
    auto, name = run("auto", [small, large])
    assert name == "tma_narrow"                 # of the group with the most points
    direct, _ = run("direct", [small])
    narrow, _ = run("tma_narrow", [large])
    for a, b in zip(auto, direct + narrow):
        assert np.array_equal(a, b)

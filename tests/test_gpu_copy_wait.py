"""Copies of the sweep that do not arrive: its CTAs record it, the loading threads load nothing more into slots they
have not seen filled, what is in flight lands before a CTA leaves, and the handle goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N", [8, 24, 41])
def test_a_lost_copy_stops_the_loads(case_dir, N, precision):
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    d = case_dir("tiny", xsplit=(0, 6, 54, 6, 0), ysplit=(0, 6, 27), zsplit=(0, 4, N - 4))
    rng = np.random.default_rng(N)
    with Simulation(d, precision=precision) as sim:
        ref = sim.run(0)
        sim.begin(0)
        sim.advance(20)
        start = {}
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            sim.set(n, rng.standard_normal(sim.get(n).shape))
            start[n] = sim.get(n)
        assert sim.selftest_copy_wait() == (True, 0)
        for n, v in start.items():
            np.testing.assert_array_equal(sim.get(n), v, err_msg=n)
        np.testing.assert_array_equal(sim.run(0), ref)

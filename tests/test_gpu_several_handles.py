"""Handles of different sizes on one device: what a later one needs of a kernel's shared memory does not take away
what an earlier one needs.  Traces bit for bit as alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grids(case_dir):
    """A deep grid on a large continuation plane, and a small one."""
    large = case_dir("tiny", xsplit=(0, 14, 42, 14, 0), ysplit=(0, 14, 36), zsplit=(0, 14, 56), arg1=1.2)
    return large, case_dir("tiny")


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kw", [{}, dict(top_planes=1), dict(zchunks=1), dict(serial_boundary=True)])
def test_a_smaller_survey_opened_later(case_dir, precision, kw):
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    large, small = grids(case_dir)
    ref = {}
    for d in (large, small):
        with Simulation(d, precision=precision, **kw) as sim:
            ref[d] = sim.run(0)
    with Simulation(large, precision=precision, **kw) as a, Simulation(small, precision=precision, **kw) as b:
        np.testing.assert_array_equal(a.run(0), ref[large])
        np.testing.assert_array_equal(b.run(0), ref[small])


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("persistent", [False, True])
def test_a_smaller_batch_opened_later(case_dir, precision, persistent):
    from tcsem_fdtd_gb300 import Batch, build

    build.build()
    large, small = grids(case_dir)

    def finish(b, slot):
        while b.stats()["running"]:
            b.advance(64)
        return b.traces(slot)

    ref = {}
    for d in (large, small):
        with Batch(precision=precision, persistent=persistent) as b:
            ref[d] = finish(b, b.add(d))
    with Batch(precision=precision, persistent=persistent) as a, Batch(precision=precision, persistent=persistent) as b:
        qa, qb = a.add(large), b.add(small)
        a.advance(2)
        b.advance(2)
        np.testing.assert_array_equal(finish(a, qa), ref[large])
        np.testing.assert_array_equal(finish(b, qb), ref[small])

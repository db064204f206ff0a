"""A batch whose slots are swept in one chunk runs its steps in pieces (few tiles: one sweep CTA per SM; more:
as they fit) or, with many tiles, in two groups of slots.  Every slot's traces against its own run in one chunk,
with the tolerances of the batch tests (FP64 1e-12, FP32 1e-6 of each trace's peak)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {64: 1e-12, 32: 1e-6}


def rel_err(got, exp):
    peak = np.abs(exp).max(axis=-1, keepdims=True)
    return float((np.abs(got - exp) / np.where(peak == 0, 1.0, peak)).max())


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("count,launches", [(1, 7), (3, 7), (7, None), (13, 12)])
def test_batch_steps_in_pieces_and_groups(case_dir, count, launches, precision):
    from tcsem_fdtd_gb300 import Batch, Simulation, build

    build.build()
    # 130 x 50 and 129 x 49 cells, 24 and 23 planes: 21 tiles each
    dirs = [case_dir("tiny", xsplit=(0, 6, 118 - q, 6, 0), ysplit=(0, 6, 38 - q), zsplit=(0, 6, 18 - q), Tn=2.5e-3, Nt=5)
            for q in (0, 1)]
    exp = []
    for d in dirs:
        with Simulation(d, precision=precision, zchunks=1) as sim:
            exp.append(sim.run(0))
    with Batch(precision=precision) as b:
        ids = [b.add(dirs[q % 2]) for q in range(count)]
        b.advance(1)
        if launches and precision == 32:
            assert b.info(ids[0])["launches_per_step"] == launches
        while b.stats()["running"]:
            b.advance(64)
        for q, s in enumerate(ids):
            e = exp[q % 2]
            assert rel_err(b.traces(s, nr=e.shape[0]), e) <= TOL[precision], (q, precision)

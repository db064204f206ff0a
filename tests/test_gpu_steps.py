"""The cooperative launch of many steps against the captured graph of the same steps.

Nine steps from random fields, in calls of one, two and six steps (either field set first), on grids whose
tiles are cut in x and y, with a single chunk and the deepest ones, an odd plane, an unfolded (padded) one, top
chunks on CTAs of their own and behind others, two frequencies per CTA and several rounds of a phase.  Each launch's FP32 fields are compared with the FP64 build's.
Tolerance: the graph's own error (times 1.5) and the rounding of the three products, sums of up to 512
terms: 3 sqrt(512) 2^-24 = 4e-6 of the array's largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Ex", "Ey", "Ez", "Bx", "By", "Bz", "BxAir", "ByAir")
ROUNDING = 4e-6


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("L,M,N,strip,growth,plane", [
    (24, 22, 20, 4, 1.2, 0), (31, 30, 9, 3, 1.1, 2), (65, 33, 25, 6, 1.2, 0), (67, 41, 24, 8, 1.2, 1),
    (200, 47, 40, 14, 1.22, 0), (98, 80, 92, 14, 1.2, 0), (135, 79, 119, 20, 1.16, 0)])
def test_cooperative_steps_against_the_graph(case_dir, L, M, N, strip, growth, plane):
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    d = case_dir("tiny", xsplit=(0, strip, L - 2 * strip, strip, 0), ysplit=(0, strip, M - 2 * strip),
                 zsplit=(0, strip, N - strip), arg1=growth)
    rng = np.random.default_rng(L)
    start, out = {}, []
    for kw in (dict(precision=64), dict(precision=32, top_planes=1), dict(precision=32)):
        with Simulation(d, padded_plane=plane, **kw) as sim:
            assert (sim.info["L"], sim.info["M"], sim.info["N"]) == (L, M, N)
            assert (sim.info["launches_per_step"] == 0) == (kw == dict(precision=32))
            sim.begin(0)
            for n in FIELDS:
                if n not in start:
                    start[n] = rng.standard_normal(sim.get(n).shape).astype(np.float32).astype(np.float64)
                sim.set(n, start[n])
            for k in (1, 2, 6):
                sim.advance(k)
            out.append({n: np.asarray(sim.get(n), np.float64) for n in FIELDS})
    exact, graph, steps = out
    for n in FIELDS:
        assert rel(steps[n], exact[n]) <= 1.5 * rel(graph[n], exact[n]) + ROUNDING, n


def test_which_grids_take_the_cooperative_launch(case_dir):
    """FP32, the default layout and order, and a small grid; everything else keeps its captured graph."""
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    d = case_dir("tiny")
    for kw, coop in ((dict(), True), (dict(graph_steps=8), True), (dict(precision=64), False), (dict(zchunks=3), False),
                     (dict(zchunks=-1), False), (dict(top_planes=2), False), (dict(serial_boundary=True), False)):
        with Simulation(d, **kw) as sim:
            assert (sim.info["launches_per_step"] == 0) == coop, kw
    # 1.6 million cells
    d = case_dir("tiny", xsplit=(0, 6, 116, 6, 0), ysplit=(0, 6, 116), zsplit=(0, 6, 90))
    with Simulation(d) as sim:
        assert sim.info["launches_per_step"] == 7


def test_states_move_between_the_launches(case_dir, tmp_path):
    """The cooperative launch keeps the chunk layout of the graph: a state either of them saved continues in the
    other one to the end of the run, and in its own bit for bit."""
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    d = case_dir("halfspace_64x64x48", Tn=2e-4, Nt=8)
    graph, coop = dict(top_planes=1), dict()
    path = str(tmp_path / "state")
    for save in (graph, coop):
        with Simulation(d, **save) as a:
            ref = a.run(0)
            a.begin(0)
            a.advance(101)
            a.save_state(path)
        for load in (graph, coop):
            with Simulation(d, **load) as b:
                assert (b.info["launches_per_step"] == 0) == (load is coop)
                b.load_state(path)
                while not b.advance(1000):
                    pass
                got = b.traces(ref.shape[0])
            assert np.isfinite(got).all()
            if load is save:
                np.testing.assert_array_equal(got, ref)

"""Grids whose marches go through more planes than the sweep's z table holds (224), or than it once held on an SM
beside another CTA's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {64: 1e-10, 32: 2e-5}  # of one step, relative to the largest magnitude: the stage tests' tolerances


def deep(case_dir, L, M, N, **kw):
    return case_dir("tiny", xsplit=(0, 6, L - 12, 6, 0), ysplit=(0, 6, M - 12), zsplit=(0, 6, N - 6), **kw)


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


# the last depth of one table, one and more planes beyond, the second refill, the deepest
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,zchunks", [(221, 1), (222, 1), (223, 1), (225, 1), (229, 2), (444, 1), (445, 1), (447, 1), (5200, 0)])
def test_fused_step_of_a_deep_march(case_dir, N, zchunks, precision):
    from oracle import oracle as orc_build
    from oracle.oracle import Oracle
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    orc_build.build()
    d = deep(case_dir, 22, 19, N)
    orc = Oracle(d)
    with Simulation(d, precision=precision, zchunks=zchunks) as sim:
        rng = np.random.default_rng(N)
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz", "BxAir", "ByAir"):
            a = rng.standard_normal(orc.field_shape(n))
            orc.set(n, a)
            sim.set(n, a)
        sched = orc.schedule()
        sim.select_tx(0)
        for step in (30, 31):
            lam, dt, wave = sched["lam"][step], sched["dt1"][step], sched["wave"][step]
            dtb = 0.5 * (dt + sched["dt2"][step])
            sim.fused_step(lam, dt, dtb, wave)
            orc.electric_field(0, lam, dt, wave)
            orc.bderivate(dtb)
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            assert rel(sim.get(n), orc.get(n)) < TOL[precision], n


@pytest.mark.parametrize("precision", [64, 32])
def test_deep_slots_of_a_batch(case_dir, precision):
    """Whole columns in pieces (all but the top plane, then that one) and through the persistent schedule, beside a
    shallow slot; one chunk alone gives the same sums.  Tolerances of the batch tests."""
    from tcsem_fdtd_gb300 import Batch, Simulation, build

    build.build()
    dirs = [deep(case_dir, 22, 19, N, Tn=1.2e-3, Nt=3) for N in (451, 40)]
    exp = []
    for d in dirs:
        with Simulation(d, precision=precision, zchunks=1) as sim:
            exp.append(sim.run(0))
    for persistent in (False, True):
        with Batch(precision=precision, persistent=persistent) as b:
            ids = [b.add(d) for d in dirs]
            while b.stats()["running"]:
                b.advance(64)
            for e, q in zip(exp, ids):
                got = b.traces(q, nr=e.shape[0])
                peak = np.abs(e).max(axis=-1, keepdims=True)
                assert float((np.abs(got - e) / np.where(peak == 0, 1.0, peak)).max()) <= {64: 1e-12, 32: 1e-6}[precision]


def test_depth_does_not_change_the_layout(case_dir):
    """Two CTAs of the FP32 sweep share an SM at any depth: as many z-chunks at 240 and 600 planes as at 160."""
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    n = []
    for N in (160, 240, 600):
        with Simulation(deep(case_dir, 128, 128, N), precision=32) as sim:
            n.append(sim.info["zchunks"])
    assert n[1] == n[0] and n[2] == n[0]


def test_states_of_both_layouts_of_a_deep_grid_continue(case_dir, tmp_path):
    """An FP32 grid of 240 planes: states in the default layout, and in the one chosen while one sweep CTA
    fitted an SM there (half the lower chunks), continue in the same handle; another layout's is refused."""
    from tcsem_fdtd_gb300 import Simulation, TcsemError, build

    build.build()
    d = deep(case_dir, 128, 128, 240, Tn=1.2e-3, Nt=3)
    ref = {}
    with Simulation(d, precision=32) as sim:
        now = sim.info["zchunks"]
        earlier = 1 + (now - 1) // 2
    for n in (now, earlier, earlier + 1):
        with Simulation(d, precision=32, zchunks=n, top_planes=1) as sim:
            ref[n] = sim.run(0)
            sim.begin(0)
            sim.advance(101)
            sim.save_state(str(tmp_path / f"s{n}"))
    with Simulation(d, precision=32) as sim:
        for n in (earlier, now, earlier):
            sim.load_state(str(tmp_path / f"s{n}"))
            while not sim.advance(1000):
                pass
            np.testing.assert_array_equal(sim.traces(ref[n].shape[0]), ref[n])
        with pytest.raises(TcsemError) as e:
            sim.load_state(str(tmp_path / f"s{earlier + 1}"))
        assert e.value.status == 3

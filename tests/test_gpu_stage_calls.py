"""The stage calls and the exchange of fields with the host where their kernels can go wrong: one plane more and
fewer than the planes a block of the Bz sum holds, cut tiles, volumes of several pieces of the exchange buffer, and
stage calls between fused steps (Bz then carries the totals of its chunks).  The oracle's stages with the tolerances
of the stage tests (FP64 1e-10, FP32 2e-5 of the largest value); values that both types hold come back unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("Ex", "Ey", "Ez", "Bx", "By", "Bz", "BxAir", "ByAir")
TOL = {64: 1e-10, 32: 2e-5}


def grid(case_dir, L, M, N, strip=6):
    return case_dir("tiny", xsplit=(0, strip, L - 2 * strip, strip, 0), ysplit=(0, strip, M - 2 * strip), zsplit=(0, strip, N - strip))


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("L,M,N", [(33, 25, 63), (32, 24, 64), (31, 23, 65), (65, 40, 130), (24, 22, 12)])
def test_stage_kernels_against_the_oracle(case_dir, L, M, N, precision):
    from oracle import oracle as orc_build
    from oracle.oracle import Oracle
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    orc_build.build()
    d = grid(case_dir, L, M, N)
    orc = Oracle(d)
    with Simulation(d, precision=precision) as sim:
        assert (sim.info["L"], sim.info["M"], sim.info["N"]) == (L, M, N)
        rng = np.random.default_rng(N)
        for n in FIELDS:
            a = rng.standard_normal(orc.field_shape(n))
            orc.set(n, a)
            sim.set(n, a)
        sched = orc.schedule()
        sim.select_tx(0)
        for step in (30, 31):
            lam, dt, wave = sched["lam"][step], sched["dt1"][step], sched["wave"][step]
            for s in (sim, orc):
                args = () if s is sim else (0,)
                s.electric_field(*args, lam, dt, wave)
                s.bderivate(0.5 * (dt + sched["dt2"][step]))
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            assert rel(sim.get(n), orc.get(n)) < TOL[precision], n


def test_stage_calls_between_fused_steps(case_dir):
    """Chunked and unchunked handles make the same mix of launches: steps, stages, a fused step, stages, a state."""
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    d = grid(case_dir, 65, 33, 40)
    got = []
    for zchunks in (1, 5):
        with Simulation(d, precision=64, zchunks=zchunks) as sim:
            sc = sim.schedule()
            sim.begin(0)
            rng = np.random.default_rng(7)
            for n in FIELDS:
                sim.set(n, rng.standard_normal(sim.field_shape(n)))

            def stages(n):
                sim.upcontinuation()
                sim.electric_field(sc["lam"][n], sc["dt1"][n], sc["wave"][n])
                sim.bderivate(0.5 * (sc["dt1"][n] + sc["dt2"][n]))

            sim.advance(3)
            stages(3)
            sim.fused_step(sc["lam"][4], sc["dt1"][4], 0.5 * (sc["dt1"][4] + sc["dt2"][4]), sc["wave"][4])
            first = sim.get("Bz")
            sim.fused_step(sc["lam"][5], sc["dt1"][5], 0.5 * (sc["dt1"][5] + sc["dt2"][5]), sc["wave"][5])
            stages(6)
            sim.advance(2)
            got.append([first] + [sim.get(n) for n in FIELDS])
    for a, b in zip(*got):
        assert rel(a, b) < 1e-10


@pytest.mark.parametrize("precision", [64, 32])
def test_fields_come_back_as_they_were_set(case_dir, precision):
    """Whole volumes in two pieces of the exchange buffer (24 planes of 290 x 310), and no other field touched."""
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    d = grid(case_dir, 290, 310, 30)
    with Simulation(d, precision=precision) as sim:
        rng = np.random.default_rng(3)
        want = {n: rng.standard_normal(sim.field_shape(n)).astype(np.float32).astype(np.float64) for n in FIELDS}
        for n in FIELDS:
            sim.set(n, want[n])
        for n in FIELDS:
            np.testing.assert_array_equal(sim.get(n), want[n])

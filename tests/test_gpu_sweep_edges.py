"""The fused sweep where its march and its tiles can go wrong: chunks of one to five planes and a whole
column (every phase of the ring the march can end in), tiles cut by the grid in x and y, one cell beyond
a whole tile, and the tile heights and chunk counts the FP64 rule chooses.  One fused step on random fields against the oracle's E stage then B stage; tolerances
of the stage tests, relative to the largest magnitude of the oracle's array (FP64 1e-10, FP32 2e-5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {64: 1e-10, 32: 2e-5}


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("L,M,N,zchunks", [(64, 40, 24, 16), (65, 33, 25, 9), (71, 36, 24, 6), (63, 39, 23, 5), (129, 32, 22, 1),
                                             (64, 64, 48, 0), (44, 38, 27, 0), (133, 45, 30, 0)])
def test_fused_step_at_tile_and_chunk_edges(case_dir, L, M, N, zchunks, precision):
    from oracle import oracle as orc_build
    from oracle.oracle import Oracle
    from tcsem_fdtd_gb300 import Simulation, build

    build.build()
    orc_build.build()
    d = case_dir("tiny", xsplit=(0, 6, L - 12, 6, 0), ysplit=(0, 6, M - 12), zsplit=(0, 6, N - 6))
    orc = Oracle(d)
    with Simulation(d, precision=precision, zchunks=zchunks) as sim:
        assert (sim.info["L"], sim.info["M"], sim.info["N"]) == (L, M, N)
        assert sim.info["zchunks"] == zchunks or zchunks == 0
        rng = np.random.default_rng(L + zchunks)
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz", "BxAir", "ByAir"):
            a = rng.standard_normal(orc.field_shape(n))
            orc.set(n, a)
            sim.set(n, a)
        sched = orc.schedule()
        sim.select_tx(0)
        for step in (30, 31):  # the second one reads the chunk-partial Bz of the first
            lam, dt, wave = sched["lam"][step], sched["dt1"][step], sched["wave"][step]
            dtb = 0.5 * (dt + sched["dt2"][step])
            sim.fused_step(lam, dt, dtb, wave)
            orc.electric_field(0, lam, dt, wave)
            orc.bderivate(dtb)
        for n in ("Ex", "Ey", "Ez", "Bx", "By", "Bz"):
            assert rel(sim.get(n), orc.get(n)) < TOL[precision], n


def test_state_of_the_earlier_default_layout_continues(case_dir, tmp_path):
    """A state saved in the layout an FP64 handle had by default before (64 x 64 x 48: six chunks, one plane
    at the top) continues in a handle with today's default layout and gives the traces of its own run; a
    state in any other layout is refused."""
    from tcsem_fdtd_gb300 import Simulation, TcsemError, build

    build.build()
    d = case_dir("halfspace_64x64x48", Tn=2e-4, Nt=8)
    with Simulation(d, precision=64) as b:
        other = next(n for n in (3, 4, 5) if n != b.info["zchunks"])
    for n, accepted in ((6, True), (other, False)):
        path = str(tmp_path / f"state{n}")
        with Simulation(d, precision=64, zchunks=n) as a:
            ref = a.run(0)
            a.begin(0)
            a.advance(101)
            a.save_state(path)
        with Simulation(d, precision=64) as b:
            if not accepted:
                with pytest.raises(TcsemError) as e:
                    b.load_state(path)
                assert e.value.status == 3
                continue
            b.load_state(path)
            while not b.advance(1000):
                pass
            np.testing.assert_allclose(b.traces(15), ref[:15], rtol=0, atol=1e-12 * np.abs(ref).max())

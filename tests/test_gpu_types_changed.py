"""Particle types that the caller replaces between a sort and the stage that
reads them (set_field("flag"), or an upload of the same particles): the stages
go by the types as they are, in the cell ranges of the last sort, as the oracle
does. Bit for bit."""
import numpy as np
import pytest

from parity_util import compare, make_pair, transplant

pytestmark = pytest.mark.gpu

CHANGES = ["air to fluid", "fluid to air", "any"]
STAGE_FIELDS = ["lsfluid", "lsair", "lsmerge", "mark", "airux", "airuy", "airuz", "waterux"]


def _changed(mp, flag, pos, change):
    flag, rng = flag.copy(), np.random.default_rng(1)
    if change == "air to fluid":
        flag[flag == mp.TYPEAIR] = mp.TYPEFLUID
    elif change == "fluid to air":
        flag[(pos[:, 0] > 0.6) & (flag == mp.TYPEFLUID)] = mp.TYPEAIR
    else:
        some = rng.random(len(flag)) < 0.05
        flag[some] = rng.choice([mp.TYPEFLUID, mp.TYPEAIR, mp.TYPEAIRSOLO, mp.TYPESOLID], some.sum())
    return flag


@pytest.mark.parametrize("change", CHANGES)
@pytest.mark.parametrize("how", ["set_field", "upload"])
def test_stages_after_types_change(mp, oracle_mod, change, how):
    sim, orc = make_pair(mp, oracle_mod, 1, 32, 11)
    sim.hashAndSortParticles()
    parts = sim.download_particles()
    parts["flag"] = _changed(mp, parts["flag"], parts["pos"], change)
    if how == "set_field":
        sim.set_field("flag", parts["flag"])
    else:
        sim.upload_particles(**parts)
    transplant(sim, orc)
    for stage in [("computeLevelset", 0.0), ("sweepLSAndMardGrid",), ("mapvelp2g_bubble",)]:
        for o in (sim, orc):
            getattr(o, stage[0])(*stage[1:])
        bad = compare({f: sim.get_field(f) for f in STAGE_FIELDS}, {f: orc.get_field(f) for f in STAGE_FIELDS})
        assert not bad, (stage, bad)
    sim.close()


@pytest.mark.parametrize("change", CHANGES)
def test_surfaces_after_types_change(mp, oracle_mod, change):
    sim, orc = make_pair(mp, oracle_mod, 1, 32, 11, b_run_mc=1)
    sim.hashAndSortParticles()
    transplant(sim, orc)
    sim.preMC()
    orc.preMC()
    parts = sim.download_particles()
    assert np.array_equal(parts["pos"], orc.download_particles()["pos"])
    flag = _changed(mp, parts["flag"], parts["pos"], change)
    sim.set_field("flag", flag)
    orc.set_field("flag", flag)
    for surface in (mp.MC_SOLID, mp.MC_FLUID, mp.MC_GAS):
        sim.runMC(surface)
        orc.runMC(surface)
        for g, r in zip(sim.mc_field() + sim.mc_mesh(surface), orc.mc_field() + orc.mc_mesh(surface)):
            assert np.array_equal(g, r), surface
    sim.close()


def test_sort_time_does_not_depend_on_the_types(mp):
    """The marking of the bricks that hold air costs next to nothing beside the
    sort (an atomic for every cell with air made the 2x grid's sort of a cloud of
    air take three times that of the same cloud of liquid)."""
    n = 128
    p = mp.scene_params(5, n)
    p.par_num_max, p.b_run_mc = 2000000, 1
    pos = (0.05 + 0.9 * np.random.default_rng(3).random((2000000, 3))).astype(np.float32)
    ms = {}
    for kind in (mp.TYPEFLUID, mp.TYPEAIR):
        sim = mp.Sim(p)
        sim.upload_particles(pos, np.full(len(pos), kind, np.int8), np.full(len(pos), p.m0, np.float32))
        sim.preMC()
        sim.kernel_timing(mp.KT_SORT)
        t = []
        for _ in range(7):
            sim.kernel_timing_reset()
            sim.preMC()
            t.append(sim.kernel_timing_read(mp.KT_SORT)[0])
        ms[kind] = np.median(t)
        sim.close()
    assert ms[mp.TYPEAIR] <= 1.5 * ms[mp.TYPEFLUID], ms

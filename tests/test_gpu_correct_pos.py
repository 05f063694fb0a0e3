"""The position correction's two kernels against the oracle, bit for bit:
particles that are sparse, that share their cells, that crowd a cell beyond
what can be staged, and that have moved since the sort; and the time of a
correction without a sort before it."""
import numpy as np
import pytest

from parity_util import grid_params, transplant

pytestmark = pytest.mark.gpu


def _particles(mp, shape, per_cell, seed=7):
    """Uniform in the inner part of the box, about per_cell in each cell there."""
    rng = np.random.default_rng(seed)
    box = np.array(shape) / shape[0]
    n = int(per_cell * np.prod([0.7 * s for s in shape])) + 1
    pos = box * (0.15 + 0.7 * rng.random((n, 3)))
    if per_cell > 100:      # all in a few cells
        pos = box * (0.5 + (rng.random((3000, 3)) - 0.5) * 1.6 / np.array(shape))
    return {"pos": pos.astype(np.float32), "mass": rng.uniform(0.01, 0.04, len(pos)).astype(np.float32),
            "flag": rng.choice([mp.TYPEFLUID, mp.TYPEFLUID, mp.TYPEAIR, mp.TYPEAIRSOLO, mp.TYPESOLID], len(pos)).astype(np.int8)}


@pytest.mark.parametrize("per_cell", [0.02, 1.0, 5.0, 7.0, 20.0, 1000.0])
@pytest.mark.parametrize("shape", [(16, 16, 16), (9, 21, 33)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("radius", [0.5, 1.3])
def test_positions(mp, oracle_mod, per_cell, shape, radius):
    p = grid_params(mp, 5, *shape)
    p.par_num_max, p.b_run_mc, p.correction_radius = 200000, 0, radius
    sim = mp.Sim(p)
    orc = oracle_mod.Oracle(p, mp.FIELD_ID, mp.MPState, mc_tables=mp.mc_tables())
    sim.upload_particles(**_particles(mp, shape, per_cell))
    sim.hashAndSortParticles()
    transplant(sim, orc)
    # the second and third from positions that have moved (with a radius below half
    # a cell, cells are left out by where a sorted particle lies in its own)
    for again in range(1 if radius < 0.6 else 3):
        sim.correctpos()
        orc.correctpos()
        g, r = sim.download_particles(), orc.download_particles()
        assert np.array_equal(g["pos"], r["pos"]), again
    sim.close()


def test_a_correction_without_a_sort_costs_about_the_same(mp):
    """Both take the same candidates: within a factor of two (staged ranges of
    blocks whose particles have spread took four times as long)."""
    sim = mp.Sim.from_config(3, 96, 5)
    sim.kernel_timing(mp.KT_CORRECT)
    ms = [[], []]
    for _ in range(7):
        sim.hashAndSortParticles()
        for moved in range(2):
            sim.kernel_timing_reset()
            sim.correctpos()
            ms[moved].append(sim.kernel_timing_read(mp.KT_CORRECT)[0])
    after_sort, moved = (np.median(m) for m in ms)
    assert moved <= 2 * after_sort, (moved, after_sort)
    sim.close()

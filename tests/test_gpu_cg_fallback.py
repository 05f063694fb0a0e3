"""A solve whose on-chip form cannot run is done by the passes: a launch that the
runtime refuses because its blocks do not fit the device together (the host's
error, no kernel runs), and exchanges that run out of time because a block that
they wait for was never launched (the waits end after a second). The result is
the passes' own."""
import ctypes as C
import time

import numpy as np
import pytest

from parity_util import grid_params

pytestmark = pytest.mark.gpu

STATE = ["tp", "waterux", "wateruy", "wateruz", "airux", "airuy", "airuz"]     # what a solve's call changes


def _sim(mp, n, heat=False, prec=0):
    """A box of liquid with a free surface and seeded face velocities, or an
    uneven temperature field over all cell types."""
    p = mp.default_params(n, n, n, 16)
    p.b_run_mc, p.precision, p.cg_tol_mode, p.cg_tol = 0, prec, mp.TOL_REL, 1e-6
    sim = mp.Sim(p)
    rng = np.random.default_rng(n)
    if heat:
        mark = rng.choice([mp.TYPEFLUID, mp.TYPEAIR, mp.TYPEVACUUM, mp.TYPESOLID], (n, n, n)).astype(np.int8)
    else:
        mark = np.full((n, n, n), mp.TYPEFLUID, np.int8)
        mark[:, :, int(0.8 * n):] = mp.TYPEVACUUM
    for a in range(3):
        edge = [slice(None)] * 3
        for e in (0, -1):
            edge[a] = e
            mark[tuple(edge)] = mp.TYPEBOUNDARY
    sim.set_field("mark", mark)
    sim.set_field("tp", rng.uniform(0, 100, (n, n, n)).astype(np.float32))
    sim.set_field("waterux", (0.1 * rng.standard_normal((n + 1) * n * n)).astype(np.float32))
    sim.kernel_timing(mp.KT_CG_UPDATE)
    return sim


def _solve(mp, sim, heat=False):
    """(result, whether the passes ran, iterations, seconds)"""
    before = {f: sim.get_field(f) for f in STATE}
    sim.kernel_timing_reset()
    t = time.perf_counter()
    if heat:
        sim.heatsim()
        it = sim.state().last_heat_cg_iters
    else:
        it, _, rc = sim.project_CG_bubble()
        assert rc == 0
    t = time.perf_counter() - t
    out = sim.get_field("tp" if heat else "press")
    for f, a in before.items():
        sim.set_field(f, a)
    return out, sim.kernel_timing_read(mp.KT_CG_UPDATE)[1] > 0, it, t


@pytest.mark.parametrize("kind", ["pressure", "pressure fp64", "heat"])
def test_refused_launch(mp, monkeypatch, kind):
    import torch
    n, many = 80, 160
    plan = (C.c_int32 * 5)()
    fp64 = int("fp64" in kind)
    mp.load_library().mp_internal_cg_plan(n, n, n, many, fp64, plan)
    assert plan[0] == many
    if torch.cuda.get_device_properties(0).multi_processor_count >= many:
        pytest.skip("the device takes as many blocks")
    heat = kind == "heat"
    monkeypatch.setenv("MP_CG_KERNEL", "tma")
    ref = _sim(mp, n, heat, fp64)
    want = _solve(mp, ref, heat)
    assert want[1] and want[0].any()
    ref.close()
    monkeypatch.delenv("MP_CG_KERNEL")
    sim = _sim(mp, n, heat, fp64)
    on_chip = _solve(mp, sim, heat)
    assert not on_chip[1]
    assert mp.load_library().mp_internal_cg_setup(sim.ctx, many, 1, 0) == 0
    for _ in range(2):
        got = _solve(mp, sim, heat)
        assert got[1] and got[2] == want[2] and np.array_equal(got[0], want[0])
    # the device's own number of SMs again
    assert mp.load_library().mp_internal_cg_setup(sim.ctx, 0, 1, 0) == 0
    got = _solve(mp, sim, heat)
    assert not got[1] and np.array_equal(got[0], on_chip[0])
    sim.close()


def test_exchange_out_of_time(mp, monkeypatch):
    n = 32
    monkeypatch.setenv("MP_CG_KERNEL", "tma")
    ref = _sim(mp, n)
    want = _solve(mp, ref)
    ref.close()
    monkeypatch.delenv("MP_CG_KERNEL")
    sim = _sim(mp, n)
    assert not _solve(mp, sim)[1]
    assert mp.load_library().mp_internal_cg_setup(sim.ctx, 0, 1, 1) == 0
    first, second = _solve(mp, sim), _solve(mp, sim)
    for got in (first, second):
        assert got[1] and got[2] == want[2] and np.array_equal(got[0], want[0])
    assert first[3] < 10 and second[3] < 0.5       # waited once, not again
    sim.close()

"""Every build of the on-chip CG kernel (groups a thread, FP32 and FP64 vectors,
one exchange an iteration or two) against the passes on the same state. A plan
for a few SMs takes a small grid through a kernel that large grids take; the
table says which, and a CPU test that the plans are those and that no build is
missing. The same for the heat matrix, whose diagonal goes by cell type, and
for its TMA and float4 passes by name, which large grids run.

All forms write the same vectors but for the order in which their FP64 dot
products add, so an FP32 alpha or beta may round the other way once in a while:
the iterations agree within one and the results within the 1e-5 that the stop
rule leaves; FP64 solves to 1e-10 agree within one rounding of the FP32 fields
that they are stored in."""
import ctypes as C
import threading

import numpy as np
import pytest

from parity_util import grid_params, rel_err

# shape, SMs (0: all 148), FP64 -> groups a thread, one exchange
PLANS = [((20, 26, 37), 16, 0, 1, 1), ((20, 26, 37), 6, 0, 2, 1), ((24, 20, 30), 3, 0, 3, 1), ((20, 26, 37), 3, 0, 4, 1),
         ((20, 26, 37), 2, 0, 6, 0), ((40, 24, 48), 3, 0, 8, 0),
         ((24, 20, 30), 20, 1, 1, 0), ((20, 26, 37), 16, 1, 2, 0), ((20, 26, 37), 8, 1, 3, 0), ((20, 26, 37), 6, 1, 4, 0),
         ((20, 26, 37), 4, 1, 6, 0), ((40, 24, 48), 6, 1, 8, 0),
         # sizes in use, on all SMs
         ((64, 64, 64), 0, 0, 1, 1), ((72, 72, 72), 0, 0, 2, 1), ((96, 80, 104), 0, 0, 3, 1), ((100, 100, 100), 0, 0, 4, 1),
         ((64, 64, 64), 0, 1, 2, 0), ((72, 72, 72), 0, 1, 3, 0), ((80, 80, 80), 0, 1, 4, 0), ((100, 100, 100), 0, 1, 8, 0)]
IDS = ["%dx%dx%d-%s-%s" % (*s, n or "all", "fp64" if d else "fp32") for s, n, d, _, _ in PLANS]


def _plan(mp, shape, sms, fp64):
    out = (C.c_int32 * 5)()
    assert mp.load_library().mp_internal_cg_plan(*shape, sms or 148, fp64, out) == 0
    return out[0], out[1], out[2]


def test_plans_cover_every_build(mp):
    for shape, sms, fp64, q, one in PLANS:
        blocks, got_q, got_one = _plan(mp, shape, sms, fp64)
        assert 0 < blocks <= (sms or 148) and (got_q, got_one) == (q, one), (shape, sms, fp64)
    built = {(0, q, 1) for q in (1, 2, 3, 4)} | {(0, q, 0) for q in (6, 8)} | {(1, q, 0) for q in (1, 2, 3, 4, 6, 8)}
    assert {(d, q, one) for _, _, d, q, one in PLANS} == built


def _marks(mp, shape, rng, types):
    mark = rng.choice(types, shape).astype(np.int8)
    nx, ny, nz = shape
    mark[:, :, int(0.75 * nz):] = mp.TYPEVACUUM
    mark[nx // 2, ny // 2, 2:nz // 2] = mp.TYPEBOUNDARY          # a pillar inside
    for a in range(3):
        edge = [slice(None)] * 3
        for e in (0, -1):
            edge[a] = e
            mark[tuple(edge)] = mp.TYPEBOUNDARY
    return mark


def _sim(mp, monkeypatch, kernel, shape, sms, fp64, heat=False, boil=False, epoch=1):
    monkeypatch.setenv("MP_CG_KERNEL", kernel)
    p = grid_params(mp, 5, *[max(s, 16) for s in shape])
    p.nx, p.ny, p.nz = shape
    p.par_num_max, p.b_run_mc, p.precision, p.cg_max_iter = 16, 0, fp64, 20000
    p.cg_tol_mode, p.cg_tol = mp.TOL_REL, 1e-10 if fp64 else 1e-6
    if heat:
        p.scene = mp.SCENE_BOILING if boil else mp.SCENE_HEATTRANSFER
        p.heatalpha_fluid, p.heatalpha_air, p.heatalpha_solid, p.heatalpha_vacuum = 0.0001, 0.005, 0.015, 0.05
    sim = mp.Sim(p)
    if not kernel:
        assert mp.load_library().mp_internal_cg_setup(sim.ctx, sms, C.c_uint32(epoch), 0) == 0
    rng = np.random.default_rng(sum(shape))
    types = [mp.TYPEFLUID, mp.TYPEAIR, mp.TYPESOLID] if heat else [mp.TYPEFLUID] * 9 + [mp.TYPEAIR]
    mark = _marks(mp, shape, rng, types)
    sim.set_field("mark", mark)
    sim.set_field("lsmerge", np.where(mark == mp.TYPEAIR, 0.5, -0.5).astype(np.float32) * np.float32(p.cellsize))
    sim.set_field("tp", (100 * rng.random(shape)).astype(np.float32))
    return sim, rng


def _faces(sim, shape, rng):
    for ax, f in enumerate(("ux", "uy", "uz")):
        d = list(shape)
        d[ax] += 1
        u = (0.1 * rng.standard_normal(d)).astype(np.float32)
        sim.set_field("water" + f, u)
        sim.set_field("air" + f, u)


def _project(mp, monkeypatch, kernel, shape, sms, fp64):
    sim, rng = _sim(mp, monkeypatch, kernel, shape, sms, fp64)
    _faces(sim, shape, rng)
    sim.kernel_timing(mp.KT_CG_UPDATE)
    it, _, rc = sim.project_CG_bubble()
    out = it, rc, sim.get_field("press"), sim.get_field("wateruz"), sim.kernel_timing_read(mp.KT_CG_UPDATE)[1]
    sim.close()
    return out


def _heat(mp, monkeypatch, kernel, shape, sms, fp64, boil):
    sim, _ = _sim(mp, monkeypatch, kernel, shape, sms, fp64, True, boil)
    sim.kernel_timing(mp.KT_CG_UPDATE)
    it = []
    for _ in range(2):
        sim.heatsim()
        it.append(sim.state().last_heat_cg_iters)
    out = it, sim.get_field("tp"), sim.kernel_timing_read(mp.KT_CG_UPDATE)[1]
    sim.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("shape,sms,fp64,q,one", PLANS, ids=IDS)
def test_pressure(mp, monkeypatch, shape, sms, fp64, q, one):
    a = _project(mp, monkeypatch, "v4", shape, sms, fp64)
    b = _project(mp, monkeypatch, "", shape, sms, fp64)
    assert a[1] == b[1] == 0 and a[4] > 0 and b[4] == 0
    assert abs(a[0] - b[0]) <= 1, (a[0], b[0])
    bound = 2.0 ** -23 if fp64 else 1e-5
    assert rel_err(b[2], a[2]) <= bound and rel_err(b[3], a[3]) <= bound


@pytest.mark.gpu
@pytest.mark.parametrize("boil", [False, True], ids=["heat", "boil"])
@pytest.mark.parametrize("shape,sms,fp64,q,one", PLANS, ids=IDS)
def test_heat(mp, monkeypatch, shape, sms, fp64, q, one, boil):
    a = _heat(mp, monkeypatch, "v4", shape, sms, fp64, boil)
    b = _heat(mp, monkeypatch, "", shape, sms, fp64, boil)
    assert a[2] > 0 and b[2] == 0 and min(a[0]) > 2
    assert max(abs(x - y) for x, y in zip(a[0], b[0])) <= 1, (a[0], b[0])
    assert rel_err(b[1], a[1]) <= 1e-5


# the passes by name: TMA tiles partial along j and k, one plane chunk and many,
# a row of one group; k-rows that split into groups of four only; and neither
@pytest.mark.gpu
@pytest.mark.parametrize("boil", [False, True], ids=["heat", "boil"])
@pytest.mark.parametrize("kernel,shape", [("tma", (40, 24, 48)), ("tma", (64, 64, 64)), ("tma", (9, 17, 16)), ("tma", (170, 20, 80)),
                                          ("v4", (40, 24, 48)), ("v4", (33, 18, 36)), ("v4", (21, 30, 47))],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_heat_passes_by_name(mp, monkeypatch, kernel, shape, boil):
    a = _heat(mp, monkeypatch, kernel, shape, 0, 0, boil)
    b = _heat(mp, monkeypatch, "", shape, 0, 0, boil)
    assert a[2] > 0 and b[2] == 0 and min(a[0]) > 2
    assert max(abs(x - y) for x, y in zip(a[0], b[0])) <= 1, (a[0], b[0])
    assert rel_err(a[1], b[1]) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("fp64", [0, 1], ids=["fp32", "fp64"])
def test_tags_near_their_end(mp, monkeypatch, fp64):
    """Tags run on from solve to solve; the exchange buffer is cleared and they
    start over before a solve's could pass 2^32 - 1: the solves up to, across and
    after that point are those of a fresh context."""
    shape, cap = (20, 26, 37), 40
    last = 2 ** 32 - 1 - 2 * cap - 8          # the highest tag that a solve of `cap` iterations may start from
    out = []
    for epoch in (1, last, last + 1):
        sim, rng = _sim(mp, monkeypatch, "", shape, 6, fp64, epoch=epoch)
        p = sim.get_params()
        p.cg_max_iter = cap
        sim.set_params(p)
        runs = []
        for _ in range(4):
            _faces(sim, shape, np.random.default_rng(2))
            with pytest.warns(RuntimeWarning):
                it, _, rc = sim.project_CG_bubble()
            assert it == cap and rc == mp.MP_ERR_NOCONVERGE
            runs.append(sim.get_field("press"))
        out.append(runs)
        sim.close()
    for runs in out:
        for press in runs:
            assert np.array_equal(press, out[0][0])


@pytest.mark.gpu
def test_contexts_on_threads(mp, monkeypatch):
    """Several contexts solve on chip at a time, each on its own thread and stream:
    every result is that of the solve alone."""
    shapes = [(32, 32, 32), (64, 64, 64), (48, 40, 56), (96, 96, 96)]
    sims, want = [], []
    for shape in shapes:
        sim, rng = _sim(mp, monkeypatch, "", shape, 0, 0)
        sims.append(sim)
        _faces(sim, shape, np.random.default_rng(4))
        sim.project_CG_bubble()
        want.append(sim.get_field("press"))
    errors = []

    def work(k):
        for _ in range(6):
            _faces(sims[k], shapes[k], np.random.default_rng(4))
            sims[k].project_CG_bubble()
            if not np.array_equal(sims[k].get_field("press"), want[k]):
                errors.append(shapes[k])

    for s in sims:
        s.kernel_timing(mp.KT_CG_UPDATE)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sims))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors and not any(t.is_alive() for t in threads)
    for s in sims:
        assert s.kernel_timing_read(mp.KT_CG_UPDATE)[1] == 0
        s.close()

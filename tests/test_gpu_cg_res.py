"""The on-chip CG solve (one cooperative launch, vectors in shared memory and
registers) against the one-launch-per-pass forms on the same state.

Both write the same vectors; only their FP64 dot products add in another
order, so an FP32-vector solve may round alpha or beta the other way once in
a while: the iteration count agrees within one and the pressure within the
1e-5 that the stop rule (relative residual 1e-6) leaves. The FP64 solves stop
at 1e-10 and agree far below FP32's spacing; pressure and faces are stored in
FP32, so they agree within one of its roundings (2^-23)."""
import numpy as np
import pytest

from parity_util import grid_params, rel_err

pytestmark = pytest.mark.gpu

# units of 32 cells: rows of one, a partial and several units; one k-row per
# tile to the largest tiles; partial tiles along i and j; a grid whose one
# axis is too short for more than one tile; the largest FP32 grids
SHAPES = [(8, 8, 8), (32, 32, 32), (32, 24, 30), (40, 24, 48), (17, 90, 65), (90, 66, 110), (200, 12, 33),
          (128, 128, 128), (60, 60, 400)]


def _project(mp, monkeypatch, kernel, shape, prec, tol, water=False):
    monkeypatch.setenv("MP_CG_KERNEL", kernel)
    p = grid_params(mp, 5, *shape)
    p.par_num_max, p.b_run_mc, p.precision, p.cg_tol, p.cg_max_iter = 16, 0, prec, tol, 20000
    sim = mp.Sim(p)
    rng = np.random.default_rng(sum(shape))
    nx, ny, nz = shape
    mark = np.full(shape, mp.TYPEFLUID, np.int8)
    mark[rng.random(shape) < 0.05] = mp.TYPEAIR
    mark[:, :, int(0.75 * nz):] = mp.TYPEVACUUM
    mark[nx // 2, ny // 2, 2:nz // 2] = mp.TYPEBOUNDARY          # a pillar inside
    for a in range(3):
        edge = [slice(None)] * 3
        for e in (0, -1):
            edge[a] = e
            mark[tuple(edge)] = mp.TYPEBOUNDARY
    sim.set_field("mark", mark)
    sim.set_field("lsmerge", np.where(mark == mp.TYPEAIR, 0.5, -0.5).astype(np.float32) * np.float32(p.cellsize))
    for ax, f in enumerate(("ux", "uy", "uz")):
        d = list(shape)
        d[ax] += 1
        u = (0.1 * rng.standard_normal(d)).astype(np.float32)
        sim.set_field("water" + f, u)
        sim.set_field("air" + f, u)
    l0 = sim.launch_count()
    it, _, rc = sim.project_CG() if water else sim.project_CG_bubble()
    out = it, rc, sim.get_field("press"), sim.get_field("wateruz"), sim.launch_count() - l0
    sim.close()
    return out


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("form", ["mixed", "water", "fp64"])
def test_on_chip_solve_equals_the_passes(mp, monkeypatch, shape, form):
    prec, tol = (mp.PREC_FP64, 1e-10) if form == "fp64" else (mp.PREC_MIXED, 1e-6)
    a = _project(mp, monkeypatch, "v4", shape, prec, tol, form == "water")
    b = _project(mp, monkeypatch, "", shape, prec, tol, form == "water")
    assert a[1] == b[1] == 0
    assert abs(a[0] - b[0]) <= 1, (a[0], b[0])
    bound = 2.0 ** -23 if form == "fp64" else 1e-5
    assert rel_err(b[2], a[2]) <= bound and rel_err(b[3], a[3]) <= bound
    if form != "fp64" or np.prod(shape) < 1000000:   # 1.4M cells and more do not fit on chip in FP64
        assert b[4] < 8, b[4]


# the TMA passes by name (grids of these sizes take the on-chip solve): partial
# tiles along j and k, one plane chunk and many, a row of one group
@pytest.mark.parametrize("shape", [(40, 24, 48), (64, 64, 64), (9, 17, 16), (170, 20, 80)],
                         ids=lambda s: "x".join(map(str, s)))
def test_tma_passes_equal_the_float4_passes(mp, monkeypatch, shape):
    a = _project(mp, monkeypatch, "v4", shape, mp.PREC_MIXED, 1e-6)
    b = _project(mp, monkeypatch, "tma", shape, mp.PREC_MIXED, 1e-6)
    assert a[1] == b[1] == 0
    assert abs(a[0] - b[0]) <= 1, (a[0], b[0])
    assert rel_err(b[2], a[2]) <= 1e-5 and rel_err(b[3], a[3]) <= 1e-5
    assert b[4] > 8, b[4]


def test_iteration_cap_and_empty_right_hand_side(mp, monkeypatch):
    """The cap stops after exactly that many iterations with the warning code;
    a zero right-hand side needs none."""
    monkeypatch.setenv("MP_CG_KERNEL", "")
    p = grid_params(mp, 5, 32, 32, 32)
    p.par_num_max, p.b_run_mc, p.cg_max_iter = 16, 0, 7
    sim = mp.Sim(p)
    mark = np.full((32, 32, 32), mp.TYPEBOUNDARY, np.int8)
    mark[1:-1, 1:-1, 1:-1] = mp.TYPEFLUID
    mark[1:-1, 1:-1, 20:-1] = mp.TYPEVACUUM
    sim.set_field("mark", mark)
    it, _, rc = sim.project_CG_bubble()
    assert (it, rc) == (0, 0) and not sim.get_field("press").any()
    u = np.random.default_rng(3).standard_normal(33 * 32 * 32).astype(np.float32)
    sim.set_field("waterux", u)
    with pytest.warns(RuntimeWarning):
        it, _, rc = sim.project_CG_bubble()
    assert it == 7 and rc == mp.MP_ERR_NOCONVERGE
    sim.close()

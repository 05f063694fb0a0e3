"""Uneven particle sets on ragged grids, GPU against the oracle: cells that hold
none, a few or well over a thousand particles of mixed types, so that the
gathers that stage particle ranges in shared memory meet ranges that are empty,
that fill several chunks or batches, and that do not fit at all. The compared
stages run the same operations in the same order on both sides and agree bit
for bit; the heat solve agrees within the 1e-5 of its stop rule."""
import numpy as np
import pytest

from parity_util import compare, grid_params, rel_err, snapshot, transplant

pytestmark = pytest.mark.gpu

SHAPES = [(17, 9, 41), (12, 23, 34), (9, 8, 96)]


def _piles(mp, shape, scale, seed, types):
    """Particles of `types` for a grid of cells of 1/nx * scale."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = shape
    cnt = rng.poisson(rng.choice([0.0, 0.3, 4.0, 9.0], size=shape))
    cnt[:, :, int(0.8 * nz):] = 0
    a, b, c = nx // 2, ny // 2, nz // 3
    cnt[a, b, c] = 1600                      # one cell beyond every staged range
    cnt[a - 1:a + 2, b + 2, c + 4] = 500     # columns that fit alone, not together
    cnt[2, 2, 5:9] = 130                     # a run of full cells
    cnt[1, 1, 1] = 300                       # next to three walls
    cell = np.repeat(np.arange(cnt.size), cnt.ravel())
    ijk = np.stack(np.unravel_index(cell, shape), 1)
    rng.shuffle(ijk)
    pos = (ijk + 0.5 + 0.98 * (rng.random(ijk.shape) - 0.5)) / nx * scale
    pos[:2] = -0.3 * scale                   # outside the grid
    n = len(pos)
    # mixed in some planes, pure in others
    flag = rng.choice(types, size=n)
    pure = ijk[:, 0] % 3 == 0
    flag[pure] = np.asarray(types)[(ijk[pure, 1] // 2) % len(types)]
    return {"pos": pos.astype(np.float32), "flag": flag.astype(np.int8),
            "mass": rng.uniform(0.01, 0.04, n).astype(np.float32),
            "vel": rng.standard_normal((n, 3)).astype(np.float32),
            "temp": rng.uniform(250, 370, n).astype(np.float32), "lheat": rng.uniform(0, 10, n).astype(np.float32),
            "solubility": rng.uniform(0, 0.02, n).astype(np.float32), "gascontain": rng.uniform(0, 0.01, n).astype(np.float32)}


def _pair(mp, oracle_mod, shape, scale=1.0, seed=5, types=None, tables=None, **overrides):
    p = grid_params(mp, 5, *shape)
    p.cellsize *= scale
    p.samplespace *= scale
    p.pradius *= scale
    p.par_num_max = 200000
    for k, v in overrides.items():
        setattr(p, k, v)
    sim = mp.Sim(p)
    orc = oracle_mod.Oracle(p, mp.FIELD_ID, mp.MPState, mc_tables=tables or mp.mc_tables())
    if tables:
        sim.set_mc_tables(*tables)
    parts = _piles(mp, shape, scale, seed, types or [mp.TYPEFLUID, mp.TYPEFLUID, mp.TYPEAIR, mp.TYPEAIRSOLO, mp.TYPESOLID])
    sim.upload_particles(**parts)
    sim.hashAndSortParticles()
    transplant(sim, orc)
    return sim, orc


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("radius", [0.5, 1.3])
def test_stages(mp, oracle_mod, shape, radius):
    sim, orc = _pair(mp, oracle_mod, shape, correction_radius=radius)
    for stage, *args in [("computeLevelset", 0.0), ("sweepLSAndMardGrid",), ("mapvelp2g_bubble",), ("correctpos",),
                         ("hashAndSortParticles",), ("computeLevelset", 0.15), ("sweepLSAndMardGrid",)]:
        getattr(sim, stage)(*args)
        getattr(orc, stage)(*args)
        bad = compare(snapshot(sim), snapshot(orc))
        assert not bad, (stage, bad)
    sim.close()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_heat(mp, oracle_mod, shape):
    sim, orc = _pair(mp, oracle_mod, shape)
    for o in (sim, orc):
        o.computeLevelset(0.0)
        o.sweepLSAndMardGrid()
        o.updateTemperature()
    for f in ("tp", "tp_save"):
        assert rel_err(sim.get_field(f), orc.get_field(f)) <= 1e-5, f
    assert rel_err(sim.download_particles()["temp"], orc.download_particles()["temp"]) <= 1e-5
    sim.close()


def _no_last_triangle(mp):
    """The tables without the last triangle of every case that has several:
    crossed edges that no triangle uses get no vertex."""
    nv, tri, _ = mp.mc_tables()
    nv, tri = nv.copy(), tri.reshape(256, 16).copy()
    for c in range(256):
        if nv[c] > 3:
            nv[c] -= 3
            tri[c, nv[c]:] = tri[0, 0]       # as behind every case's last vertex
    return nv, tri.reshape(-1)


@pytest.mark.parametrize("case", ["17x9x41", "12x23x34", "9x8x96", "fine scale", "no gas", "gas alone", "tables"])
def test_surfaces(mp, oracle_mod, case):
    kw = {}
    shape = (12, 23, 34)
    if "x" in case:
        shape = tuple(map(int, case.split("x")))
    elif case == "fine scale":
        kw["scale"] = 2.0 ** -15             # the density's general square root
    elif case == "no gas":
        kw["types"] = [mp.TYPEFLUID, mp.TYPESOLID]
    elif case == "gas alone":
        kw["types"] = [mp.TYPEAIR, mp.TYPEAIRSOLO]
    else:
        kw["tables"] = _no_last_triangle(mp)
    sim, orc = _pair(mp, oracle_mod, shape, **kw)
    sim.preMC()
    orc.preMC()
    verts = 0
    for surf in (mp.MC_SOLID, mp.MC_FLUID, mp.MC_GAS):
        sim.runMC(surf)
        orc.runMC(surf)
        (gd, gc), (rd, rc) = sim.mc_field(), orc.mc_field()
        assert np.array_equal(gd, rd) and np.array_equal(gc, rc), surf
        for g, r in zip(sim.mc_mesh(surf), orc.mc_mesh(surf)):
            assert g.shape == r.shape and np.array_equal(g, r), surf
            verts += len(g)
    assert verts
    sim.close()


@pytest.mark.parametrize("shape", [(17, 9, 41), (16, 16, 40)], ids=lambda s: "x".join(map(str, s)))
def test_adjoint(mp, shape):
    """The replay ends where the engine does, bit for bit, and the FP64 adjoint
    agrees with central differences along velocity directions (1e-5: the
    differences' own error at a step of 1e-7, which crosses no kink)."""
    import torch
    p = grid_params(mp, 1, *shape)
    p.b_correct_position = 0
    p.par_num_max = 200000
    sim = mp.Sim(p)
    parts = _piles(mp, shape, 1.0, 9, [mp.TYPEFLUID, mp.TYPEFLUID, mp.TYPEAIR])
    parts["pos"][:2] = parts["pos"][2:4]
    parts["mass"][:] = p.m0
    sim.upload_particles(**{k: parts[k] for k in ("pos", "flag", "mass", "vel")})
    parts = sim.download_particles()
    x0 = torch.from_numpy(parts["pos"].astype(np.float64)).cuda()
    v0 = torch.from_numpy(0.1 * parts["vel"].astype(np.float64)).cuda()
    v0 = v0.float().double()
    sim.upload_particles(pos=parts["pos"], flag=parts["flag"], mass=parts["mass"], vel=v0.cpu().numpy())
    sim.adj_record(2, 1)
    after = sim.download_particles()
    ids = sim.adj_order().cpu().numpy()
    xT, vT = (t.cpu().numpy().astype(np.float32) for t in sim.adj_forward(x0, v0, mp.PREC_MIXED))
    assert np.array_equal(xT[ids], after["pos"]) and np.array_equal(vT[ids], after["vel"])
    gen = torch.Generator(device="cpu").manual_seed(5)
    w = [torch.randn(x0.shape, generator=gen, dtype=torch.float64).cuda() for _ in range(4)]
    _, vb = sim.step_adjoint(x0, v0, w[0], w[1], mp.PREC_FP64)

    def f(v):
        a, b = sim.adj_forward(x0, v, mp.PREC_FP64)
        return float((a * w[0]).sum() + (b * w[1]).sum())

    for d in w[2:]:
        eps = 1e-7
        fd, ad = (f(v0 + eps * d) - f(v0 - eps * d)) / (2 * eps), float((vb * d).sum())
        assert abs(fd - ad) <= 1e-5 * max(abs(fd), abs(ad)), (fd, ad)
    sim.close()

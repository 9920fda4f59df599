"""The native engine's pair list (csrc/pairs.cu): what the two spheres of a pair
hold mirrors one another through rebuilds, a list entry without its mirror image
(a slot overflow) acts on its own sphere alone, and sizes at the edges of the
kernels' blocks give the lists and forces of the FP64 path."""
import copy

import numpy as np
import pytest

import _workloads
from gpucode_gb300 import _abi
from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _by_pair(counts, partners, rec, brg):
    """(i, j) -> (record, flag) of every list entry"""
    out = {}
    for i in range(len(counts)):
        for a in range(counts[i]):
            out[(i, int(partners[i, a]))] = (rec[i, a], int(brg[i, a]))
    return out


@pytest.mark.parametrize("make", [_workloads.small_dry, _workloads.small_wet])
def test_the_two_sides_of_a_pair_mirror_one_another(cuda, make):
    """after steps with several rebuilds (every rebuild turns some pairs round),
    both spheres of every pair report the same contact, the spring negated"""
    w = make()
    pos, vel, ang = _workloads.stirred(w)
    e = Engine(w.setup, precision="mixed")
    e.set_state(pos, vel, ang)
    e.step(150)
    e.sync()
    assert e.stats()["rebuilds"] >= 2
    n, p = e.neighbors()
    rec, brg = e.history(int(n.max()))
    e.close()
    d = _by_pair(n, p, rec, brg)
    held = 0
    for (i, j), (r, b) in d.items():
        r2, b2 = d[(j, i)]  # every entry has its mirror image
        np.testing.assert_array_equal(r[:3], -r2[:3])
        np.testing.assert_array_equal(r[3:], r2[3:])
        assert b == b2
        held += bool(r[7])
    assert held > 100


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_entry_without_mirror_image_acts_on_its_own_sphere(cuda, precision):
    """lists cut at capacity: some spheres list a partner that does not list
    them.  From rest the first step's force on a sphere is gravity, the Hertz
    (or plastic) forces of the partners it lists and the walls' -- checked on
    the spheres away from the walls, one-sided entries included"""
    w = _workloads.small_dry()
    setup = copy.deepcopy(w.setup)
    full = Engine(w.setup, precision="fp64")
    pos, _, _ = _workloads.stirred(w)
    full.set_state(pos)
    full.step(1)
    full.sync()
    cap = int(full.neighbors()[0].max()) - 1
    full.close()
    setup.s.level_nnebors[0] = cap
    setup.s.n_pp_slots = cap * setup.s.level_npars[0]
    e = Engine(setup, precision=precision)
    e.set_state(pos)
    e.step(1)
    with pytest.raises(_abi.DemError) as ei:
        e.sync()
    assert ei.value.code == _abi.DEM_ERR_OVERFLOW
    n, p = e.neighbors()
    f = e.get_state()["force"]
    e.close()
    listed = {(i, int(p[i, a])) for i in range(len(n)) for a in range(n[i])}
    one_sided = [(i, j) for (i, j) in listed if (j, i) not in listed]
    assert one_sided
    s, rad = setup.s, setup.rad
    R, bw = s.cyl.R, s.cyl.Bw
    free = (np.hypot(pos[:, 0], pos[:, 1]) + rad < R) & (pos[:, 2] - rad > bw)
    want = np.zeros_like(pos)
    want[:, 2] -= (2 * rad) ** 3
    for i, j in listed:
        d = pos[i] - pos[j]
        L = np.linalg.norm(d)
        nrm = rad[i] + rad[j] - L
        if nrm <= 0:
            continue
        r = rad[i] * rad[j] / (rad[i] + rad[j])
        fn = 4 / 3 * s.cal.emod * np.sqrt(r) * nrm ** 1.5
        if nrm > s.cal.ydsp_t * r:
            fn = s.cal.yforce_t * r * r + s.cal.ystiff_t * r * (nrm - s.cal.ydsp_t * r)
        want[i] += fn * d / L
    scale = np.abs(want[free]).max()
    # FP64: the two orders of summation; mixed: the FP32 overlap and law
    tol = {"fp64": 1e-11, "mixed": 2e-5}[precision]
    assert any(free[i] for i, _ in one_sided)
    assert np.abs(f - want)[free].max() <= tol * scale


@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 128, 129, 255, 256, 257, 511, 513])
def test_lists_and_forces_at_block_edges(cuda, n):
    """the mixed engine against the FP64 one at sizes around the kernels' warps
    and blocks: the same lists, forces to the FP32 law's tolerance"""
    w = _workloads.small_wet(n=n, n_levels=1 if n < 3 else 3)
    pos, vel, ang = _workloads.stirred(w, vscale=0.05, wscale=0.1)
    got = {}
    for precision in ("fp64", "mixed"):
        e = Engine(w.setup, precision=precision)
        e.set_state(pos, vel, ang)
        e.step(1)
        e.sync()
        c, p = e.neighbors()
        got[precision] = (c, p, e.get_state()["force"], e.stats())
        e.close()
    a, b = got["fp64"], got["mixed"]
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
    assert np.abs(a[2] - b[2]).max() <= 2e-5 * np.abs(a[2]).max()
    for k in ("nb_entries", "contacts", "bridges", "wall_contacts"):
        assert a[3][k] == b[3][k], k


@pytest.mark.parametrize("levels, spread", [(1, 1.0), (4, 1.0), (4, 6.0), (3, 0.3)])
@pytest.mark.parametrize("bounded", [True, False])
def test_pruned_search_lists_what_the_full_search_lists(cuda, levels, spread, bounded):
    """The mixed engine's neighbour search skips cells no partner can reach from
    (when every radius is within its level's); the FP64 engine searches the
    reference's boxes.  The same lists, entry for entry, for spheres strewn
    through the whole computing zone and beyond its faces, equal sizes to a
    ratio of 12, and with radii above their level's (which turn the skipping
    off)."""
    from gpucode_gb300 import configs

    rng = np.random.default_rng(levels + int(10 * spread))
    n = 3000
    dia = 0.25e-3 * np.exp(np.minimum(spread, 2.5) * rng.random(n)) if levels > 1 else np.full(n, 1e-3)
    real = float(dia.max())
    inp = configs.make_input(n, levels, real, 0.1 * dia.max() / dia.min(), 4e-3, 8e-3, configs.RHO, configs.E_YOUNG,
                             configs.NU, configs.MU, 6.6e-6, configs.yldp_for_yield_overlap(0.01, 1e7, 0.3), 0,
                             dt=1e-9)
    setup = configs.Setup.build(inp, dia)
    s = setup.s
    if not bounded:
        # (the slots' counts stay the level's: a sphere too large for its level)
        big = np.flatnonzero(setup.rad > 0.9 * np.array(list(s.level_size))[setup.plevel])[::7]
        setup.rad[big] = np.array(list(s.level_size))[setup.plevel[big]] * 1.2
    lo = np.array([s.prm.Origin.x, s.prm.Origin.y, s.prm.Origin.z])
    hi = np.array([s.prm.EndPoint.x, s.prm.EndPoint.y, s.prm.EndPoint.z])
    pos = lo + (hi - lo) * rng.random((n, 3))
    pos[::50] = lo - 0.4 * rng.random((len(pos[::50]), 3))  # outside: kept in the first cells
    got = []
    for precision in ("fp64", "mixed"):
        e = Engine(setup, precision=precision)
        e.set_state(pos)
        e.step(1)
        c, p = e.neighbors(1024)
        got.append((c, p))
        e.close()
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][0].sum() > n // 4


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_longer_lists_change_no_force(cuda, precision):
    """A wider skin lists several times the partners (a warp's entries then fill
    several of the FP64 kernel's chunks) but, on the same cells, the same
    contacts in the same order: a dry bed's forces keep their bits"""
    from gpucode_gb300 import configs

    w = _workloads.small_dry()
    pos, vel, ang = _workloads.stirred(w, vscale=0.05, wscale=0.1)
    got = []
    w.inp.cut_gap = 1.5
    for skin in (0.1, 0.6, 1.5):
        setup = configs.Setup.build(w.inp, w.dia)
        setup.s.prm.SearchGap = skin
        e = Engine(setup, precision=precision)
        e.set_state(pos, vel, ang)
        e.step(1)
        e.sync()
        got.append((int(e.neighbors(512)[0].sum()), e.get_state()["force"]))
        e.close()
    assert got[2][0] * 32 / w.setup.n > 2 * 320 > got[0][0] * 32 / w.setup.n
    for _, f in got[1:]:
        np.testing.assert_array_equal(f, got[0][1])


def test_levels_side_by_side_step_every_sphere(cuda):
    """from 600,000 spheres on the sphere kernel takes its blocks level beside
    level (level sizes that are no multiples of a block): three steps give the
    FP64 engine's, forces to 2e-5 of their scale as elsewhere, and every sphere
    has moved once a step (from rest, gravity alone is 5e-7 x 9.8 of velocity a
    step in the reduced units, far above FP64's resolution)"""
    from gpucode_gb300 import configs

    w = configs.wet(n=600_053, cyl_r=0.04)
    out = {}
    for precision in ("fp64", "mixed"):
        e = Engine(w.setup, precision=precision)
        e.set_state(w.pos0_reduced)
        e.step(3)
        e.sync()
        out[precision] = e.get_state()
        e.close()
    f, g = out["fp64"], out["mixed"]
    assert (np.abs(g["vel"]).max(axis=1) > 0).all()
    np.testing.assert_allclose(g["force"], f["force"], rtol=2e-5, atol=2e-5 * np.abs(f["force"]).max())
    np.testing.assert_allclose(g["pos"], f["pos"], rtol=0, atol=1e-9)

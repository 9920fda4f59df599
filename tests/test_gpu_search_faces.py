"""The mixed engine's neighbour search in beds a few cells wide, with spheres
past the upper faces of the computing zone.  The reference's clamp hashes those
into the first cell of the next row or plane (kernel.cu:627-629), far from where
they are; a search that skips cells by their distance must still list what the
reference's boxes list."""
import numpy as np
import pytest

from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 2, 4])
@pytest.mark.parametrize("scale", [1.0, 1.4, 2.0, 3.5])
@pytest.mark.parametrize("width", [1.05, 3.3])
def test_narrow_beds_list_what_the_full_search_lists(cuda, levels, scale, width):
    """the FP64 engine searches the reference's boxes: the same lists, entry for
    entry; width: the cylinder's in largest diameters, scale: of the cells
    (dem_scale_cells)"""
    from gpucode_gb300 import configs

    rng = np.random.default_rng(int(10 * width) + levels)
    n = 400
    big = 1e-3
    dia = big * np.exp(-1.8 * rng.random(n)) if levels > 1 else np.full(n, big)
    dia[0] = big
    inp = configs.make_input(n, levels, big, 0.1 * dia.max() / dia.min(), 0.5 * width * big, 12e-3, configs.RHO,
                             configs.E_YOUNG, configs.NU, configs.MU, 6.6e-6,
                             configs.yldp_for_yield_overlap(0.01, 1e7, 0.3), 0, dt=1e-9)
    setup = configs.Setup.build(inp, dia)
    setup.scale_cells(scale)
    s = setup.s
    lo = np.array([s.prm.Origin.x, s.prm.Origin.y, s.prm.Origin.z])
    # each sphere within its own level's cells, the upper half of z empty (past
    # that face a sphere has no cell of its level)
    cells = np.array([[s.grid_size[l].x, s.grid_size[l].y, 0.5 * s.grid_size[l].z] for l in range(levels)])
    span = (cells * np.array(list(s.cell_size)[:levels])[:, None])[setup.plevel]
    pos = lo + span * rng.random((n, 3))
    for k, axes in ((0, [0]), (1, [1]), (2, [0, 1])):
        for a in axes:
            pos[k::5, a] = lo[a] + span[k::5, a] + 0.3 * rng.random(len(pos[k::5]))
    got = []
    for precision in ("fp64", "mixed"):
        e = Engine(setup, precision=precision)
        e.set_state(pos)
        e.step(1)
        got.append(e.neighbors(1024))
        e.close()
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][0].sum() > 0

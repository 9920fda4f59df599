"""The memory plan where a sphere has few neighbour slots: the arrays that go by
the sphere outweigh those that go by the slot."""
import numpy as np
import pytest

from gpucode_gb300 import configs
from gpucode_gb300.engine import Engine


def _setup(n, slots):
    """equal spheres with so many neighbour slots each"""
    inp = configs.make_input(n, 1, 1e-3, 0.1, 4e-3, 8e-3, configs.RHO, configs.E_YOUNG, configs.NU, configs.MU, 6.6e-6,
                             configs.yldp_for_yield_overlap(0.01, 1e7, 0.3), 0, dt=1e-9)
    setup = configs.Setup.build(inp, np.full(n, 1e-3))
    setup.s.level_nnebors[0] = slots
    setup.s.n_pp_slots = slots * n
    return setup


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_a_slot_more_never_needs_less(precision):
    totals = [_setup(10_000, k).memory(precision)["total"] for k in range(1, 40)]
    assert all(b > a for a, b in zip(totals, totals[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("slots", [1, 2, 4])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_estimate_covers_short_lists(cuda, precision, slots):
    """8,000,000 spheres (the plan's fixed reserve for rounding is 134 MB)"""
    import torch

    setup = _setup(8_000_000, slots)
    est = setup.memory(precision)["total"]
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    e = Engine(setup, precision=precision)
    used = free0 - torch.cuda.mem_get_info()[0]
    e.close()
    assert 0.9 * est < used <= est, (used, est)

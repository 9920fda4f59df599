"""Device-chained steps in graphs of one to eight steps (csrc/chain.cu):
calls of every length, a rebuild falling on any step of a graph, and a moving
top wall give the bits of host-driven steps."""
import copy

import numpy as np
import pytest

import _workloads
from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topv", [0.0, -5.0])
def test_calls_of_every_length_equal_host_steps(cuda, topv):
    """200-odd steps: the stirred bed rebuilds several times, at steps that fall
    differently into the graphs of each sequence of calls.  Equal bits: both
    launch the same kernels."""
    w = _workloads.small_wet()
    setup = copy.deepcopy(w.setup)
    setup.s.cyl.topv = topv
    pos, vel, ang = _workloads.stirred(w)
    total = 210
    runs = {"host": [total], "one call": [total], "rising": list(range(1, 21)),
            "odd": [1, 1, 2, 3, 3] * 21, "sevens": [7] * 30}
    out = {}
    for name, calls in runs.items():
        assert sum(calls) == total
        e = Engine(setup, precision="mixed", use_graph=name != "host")
        e.set_state(pos, vel, ang)
        for k in calls:
            e.step(k)
        e.sync()
        out[name] = (e.get_state(), e.stats()["rebuilds"])
        e.close()
    s0, r0 = out.pop("host")
    assert r0 >= 2
    for name, (s, r) in out.items():
        assert r == r0, name
        for k in ("pos", "vel", "angvel", "force"):
            assert np.array_equal(s[k], s0[k]), (name, k)

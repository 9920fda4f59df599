"""Calls that drop the captured step graphs while chained steps may still be
under way wait for those steps first."""
import numpy as np
import pytest

import _workloads
from gpucode_gb300 import _abi
from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 200])
def test_systems_set_behind_queued_steps(cuda, steps):
    """one system in the set-up's own cylinder, set right behind a call of steps
    or after waiting for them: the same bits"""
    w = _workloads.small_wet()
    pos, vel, ang = _workloads.stirred(w, vscale=0.05, wscale=0.1)
    cyl = _abi.CylinderBC.from_buffer_copy(w.setup.s.cyl)
    out = []
    for wait in (False, True):
        e = Engine(w.setup, precision="mixed")
        e.set_state(pos, vel, ang)
        e.step(steps)
        if wait:
            e.sync()
        e.set_systems(np.zeros(w.setup.n, np.int32), [cyl])
        e.step(5)
        e.sync()
        s = e.stats()
        assert s["iter"] == steps + 5 and s["error_bits"] == 0
        out.append(e.get_state())
        e.close()
    for k in ("pos", "vel", "angvel", "force"):
        np.testing.assert_array_equal(out[0][k], out[1][k])

"""The rebuild in front of the step graphs' first use: where the host knows that
one is requested it runs ahead of the graphs' building, and the bits and the
number of rebuilds are those of host-driven steps."""
import numpy as np
import pytest

import _workloads
from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu

SEQUENCES = {
    "fresh": [("step", 3)],
    "fresh, one step": [("step", 1), ("step", 1)],
    "import before the graphs of several steps": [("step", 1), ("import", 0), ("step", 5)],
    "import after them": [("step", 4), ("import", 0), ("step", 5), ("step", 1)],
    "import answered by a profile": [("import", 0), ("profile", 0), ("step", 5)],
    "loaded lists": [("save", 0), ("load", 0), ("step", 3)],
    "imported, then loaded": [("step", 2), ("save", 0), ("import", 0), ("load", 0), ("step", 3)],
    "no steps asked for": [("import", 0), ("step", 0), ("step", 2)],
}


@pytest.mark.parametrize("name", SEQUENCES)
def test_first_calls_equal_host_steps(cuda, tmp_path, name):
    w = _workloads.small_wet()
    pos, vel, ang = _workloads.stirred(w)
    out = []
    for graph in (True, False):
        e = Engine(w.setup, precision="mixed", use_graph=graph)
        e.set_state(pos, vel, ang)
        path = tmp_path / f"cp{graph}"
        for what, k in SEQUENCES[name]:
            if what == "step":
                e.step(k)
            elif what == "import":
                e.set_state(pos * 1.0001, vel, ang)
            elif what == "profile":
                e.profile_kernels()
            elif what == "save":
                e.save(path)
            else:
                e.load(path)
        e.sync()
        out.append((e.get_state(), e.stats()["rebuilds"], e.neighbors()))
        e.close()
    (a, ra, na), (b, rb, nb) = out
    assert ra == rb >= 1
    for k in ("pos", "vel", "angvel", "force"):
        np.testing.assert_array_equal(a[k], b[k])
    for x, y in zip(na, nb):
        np.testing.assert_array_equal(x, y)

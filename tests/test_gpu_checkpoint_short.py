"""Checkpoints that are refused, a load right behind queued steps, and what a file holds."""
import numpy as np
import pytest

import _workloads
from gpucode_gb300 import _abi
from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _engine(precision, steps, seed=7):
    w = _workloads.small_wet()
    pos, vel, ang = _workloads.stirred(w, seed=seed, vscale=0.2, wscale=0.5)
    e = Engine(w.setup, precision=precision)
    e.set_state(pos, vel, ang)
    e.step(steps)
    return e


def _equal(a, b):
    for k in ("pos", "vel", "angvel", "force"):
        np.testing.assert_array_equal(a[k], b[k])


@pytest.mark.parametrize("keep", [0.02, 0.5, 0.999])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_a_truncated_checkpoint_changes_nothing(cuda, tmp_path, precision, keep):
    """a file cut anywhere is an error, and the steps after it are those of an
    engine that never tried"""
    other = _engine(precision, 40, seed=8)
    other.save(tmp_path / "whole")
    other.close()
    data = (tmp_path / "whole").read_bytes()
    (tmp_path / "cut").write_bytes(data[: int(len(data) * keep)])
    out = []
    for path in ("cut", None):
        e = _engine(precision, 40)
        if path:
            with pytest.raises(_abi.DemError) as err:
                e.load(tmp_path / path)
            assert err.value.code == _abi.DEM_ERR_IO
        e.step(20)
        e.sync()
        out.append(e.get_state())
        e.close()
    _equal(*out)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_a_load_behind_queued_steps_waits_for_them(cuda, tmp_path, precision):
    """the loaded state, whatever was still under way"""
    saved = _engine(precision, 40, seed=8)
    saved.save(tmp_path / "cp")
    saved.step(10)
    want = saved.get_state()
    saved.close()
    e = _engine(precision, 300)
    e.load(tmp_path / "cp")
    e.step(10)
    got = e.get_state()
    e.close()
    _equal(got, want)


@pytest.mark.parametrize("extra", [0, 37])
def test_slots_of_no_level_are_written_too(cuda, tmp_path, extra):
    """a set-up with more slots than its levels use: the file has them all, and a
    resumed run keeps its bits"""
    w = _workloads.small_wet()
    w.setup.s.n_pp_slots += extra
    pos, vel, ang = _workloads.stirred(w, vscale=0.2, wscale=0.5)
    a, b = Engine(w.setup, precision="mixed"), Engine(w.setup, precision="mixed")
    a.set_state(pos, vel, ang)
    a.step(40)
    a.save(tmp_path / "cp")
    b.load(tmp_path / "cp")
    for e in (a, b):
        e.step(20)
        e.sync()
    _equal(a.get_state(), b.get_state())
    a.close()
    b.close()

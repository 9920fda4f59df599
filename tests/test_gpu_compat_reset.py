"""The drop-in entry points over a device reset: what the library keeps on the
device belongs to the context that is gone, and its addresses come back as the
caller's own arrays in the next.  Runs in a process of its own, without torch
(whose allocator does not survive a reset)."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


class _Array:
    """what DropInDriver uses of a device tensor, on the runtime API"""

    def __init__(self, rt, host):
        self.rt, self.host = rt, np.ascontiguousarray(host)
        self.ptr = C.c_void_p()
        assert rt.cudaMalloc(C.byref(self.ptr), C.c_size_t(max(self.host.nbytes, 1))) == 0
        self._up()

    def _up(self):
        assert self.rt.cudaMemcpy(self.ptr, self.host.ctypes.data_as(C.c_void_p), C.c_size_t(self.host.nbytes), 1) == 0

    def get(self):
        assert self.rt.cudaMemcpy(self.host.ctypes.data_as(C.c_void_p), self.ptr, C.c_size_t(self.host.nbytes), 2) == 0
        return self.host.copy()

    def data_ptr(self):
        return self.ptr.value

    def contiguous(self):
        return self

    def item(self):
        return self.get().item()

    def zero_(self):
        self.host[...] = 0
        self._up()

    def copy_(self, other):
        self.host[...] = other.get()
        self._up()


class _Arrays:
    float64, int32 = np.float64, np.int32

    def __init__(self, rt):
        self.rt = rt

    def zeros(self, *shape, dtype, device):
        return _Array(self.rt, np.zeros(shape, dtype))

    def tensor(self, x, dtype=None, device=None):
        return _Array(self.rt, np.array(x, dtype))


def _run():
    sys.path[:0] = [str(ROOT), str(ROOT / "tests")]
    import _workloads
    from gpucode_gb300 import _abi
    from gpucode_gb300.dropin import DropInDriver, declare

    lib = _abi.load()
    declare(lib)
    rt = C.CDLL("libcudart.so.13")  # the library's own
    w = _workloads.small_wet()
    pos, vel, ang = _workloads.stirred(w, vscale=0.05, wscale=0.1)
    for precision in (_abi.PREC_FP64, _abi.PREC_MIXED):
        assert lib.dem_compat_set_precision(precision) == 0
        got = []
        for _ in range(3):
            d = DropInDriver(w, pos, vel, ang, _Arrays(rt))
            for _ in range(3):
                d.step()
            got.append([v.get() for v in (d.pos, d.vel, d.force, d.lqd, d.num)])
            assert lib.dem_compat_errors() == 0
            assert rt.cudaDeviceReset() == 0
        for g in got[1:]:
            for a, b in zip(g, got[0]):
                np.testing.assert_array_equal(a, b)
    print("same bits")


@pytest.mark.gpu
def test_entry_points_after_a_device_reset(cuda):
    """three steps, a reset, the same three steps in fresh arrays: the same bits,
    in both precisions"""
    r = subprocess.run([sys.executable, __file__], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0 and "same bits" in r.stdout, r.stdout + r.stderr


if __name__ == "__main__":
    _run()

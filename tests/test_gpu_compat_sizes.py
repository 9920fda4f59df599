"""The drop-in's mixed force kernels pack the spheres, keep the slots in contact
as dense lists of 64 a warp and sift the walls in strided groups of 32: sizes at
the edges of warps and blocks, beds of one and of several levels, give the FP64
kernels' forces from the same state."""
import numpy as np
import pytest

import _workloads
from gpucode_gb300 import _abi
from gpucode_gb300.dropin import DropInDriver, declare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,n", [(_workloads.small_dry, n) for n in (2, 31, 33, 385)]
                         + [(_workloads.small_wet, n) for n in (24, 32, 97, 1153)])
def test_mixed_forces_match_fp64_from_the_same_state(cuda, make, n):
    """One step from the same stirred state.  FP32 forces from FP64 gaps: 2e-5 of
    the step's force scale, the mixed path's per-step tolerance elsewhere; the
    bridge counts are equal."""
    import torch

    lib = _abi.load()
    declare(lib)
    w = make(n)
    pos, vel, ang = _workloads.stirred(w)
    got = {}
    try:
        for name, code in (("fp64", 0), ("mixed", 1)):
            _abi.check(lib.dem_compat_set_precision(code), "dem_compat_set_precision")
            drv = DropInDriver(w, pos, vel, ang, torch)
            drv.step()
            torch.cuda.synchronize()
            got[name] = (drv.force.cpu().numpy(), drv.lqd.cpu().numpy())
    finally:
        _abi.check(lib.dem_compat_set_precision(0), "dem_compat_set_precision")
    assert lib.dem_compat_errors() == 0
    f, g = got["fp64"][0], got["mixed"][0]
    np.testing.assert_allclose(g, f, rtol=2e-5, atol=2e-5 * np.abs(f).max())
    np.testing.assert_array_equal(got["mixed"][1], got["fp64"][1])

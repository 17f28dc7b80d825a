"""Host states whose nine planes lie apart are exchanged plane by plane, consecutive ones in one copy:
both give the same state, uploaded, downloaded and in a batch."""

import ctypes as C

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200 import workloads as wl
from mhd_gpu_solver_b200.batch import BatchSolver, fixed_params
from mhd_gpu_solver_b200.mhd_solver import apply_boundary_conditions

pytestmark = pytest.mark.gpu


def _apart(state):
    """The planes of a state in nine arrays of their own, in reverse order of allocation."""
    planes = [np.array(state[c]) for c in reversed(range(9))][::-1]
    return planes, (C.POINTER(C.c_double) * 9)(
        *[p.ctypes.data_as(C.POINTER(C.c_double)) for p in planes])


@pytest.mark.parametrize("precision", [_capi.FP64, _capi.FP32])
def test_planes_apart_and_consecutive(precision):
    nx, ny = 50, 34
    U = wl.embed(wl.to_conservative(wl.fourier_state(nx, ny, 6), 5.0 / 3.0))
    apply_boundary_conditions(U, nx, ny, 2, 0, 0)
    n = U[0].size
    params = _capi.make_params(limiter=_capi.MC)
    outs = []
    for apart in (False, True):
        dev = _capi.DeviceSolver(nx, ny, precision=precision)
        try:
            dev.configure(_capi.BC_PERIODIC, _capi.BC_PERIODIC)
            if apart:
                planes, ptrs = _apart(U)
                _capi.raise_for(_capi.lib.mhdb_upload(dev.handle, ptrs, n), dev.handle)
            else:
                dev.upload(U)
            dev.solve_steps(params, 5)
            outs.append(dev.download())
            planes, ptrs = _apart(np.zeros_like(U))
            _capi.raise_for(_capi.lib.mhdb_download(dev.handle, ptrs, n), dev.handle)
            outs.append(np.stack(planes))
        finally:
            dev.close()
    for got in outs[1:]:
        assert np.array_equal(got, outs[0])

    batch = BatchSolver(precision)
    try:
        sid = batch.add(U, fixed_params(5, limiter=_capi.MC), (0, 0), fixed_steps=True)
        batch.step(5)
        whole = batch.download(sid)
        planes, ptrs = _apart(np.zeros_like(U))
        assert _capi.lib.mhdb_batch_download(batch._b, sid, ptrs, n) == _capi.OK
        assert np.array_equal(np.stack(planes), whole)
    finally:
        batch.close()

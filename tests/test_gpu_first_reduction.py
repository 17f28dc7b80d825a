"""The first signal-speed reduction of an FP32-mixed solve reads the hi planes only. Its c_h must be the
maximum over the state rounded to FP32 (the FP64 speed of the same state to FP32 rounding: 20 FP32
operations of 6e-8, held to 2e-6), alone and in a batch alike, and a state with an infinite energy
somewhere must start as it did when both planes were summed (that cell counts as NaN)."""

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200 import workloads as wl
from mhd_gpu_solver_b200.batch import BatchSolver, fixed_params
from mhd_gpu_solver_b200.mhd_solver import apply_boundary_conditions
from tests.helpers import signal_speed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("infinite", [False, True])
@pytest.mark.parametrize("nx,ny", [(1, 1), (33, 20), (200, 160)])
def test_first_c_h(nx, ny, infinite):
    U = wl.embed(wl.to_conservative(wl.fourier_state(nx, ny, 8), 5.0 / 3.0))
    if infinite:
        U[4, 2, 2] = np.inf
    apply_boundary_conditions(U, nx, ny, 2, 0, 0)
    dev = _capi.DeviceSolver(nx, ny, precision=_capi.FP32)
    try:
        dev.configure(_capi.BC_PERIODIC, _capi.BC_PERIODIC)
        dev.upload(U)
        r = dev.solve_steps(_capi.make_params(limiter=_capi.MC), 1)
    finally:
        dev.close()
    batch = BatchSolver(_capi.FP32)
    try:
        sid = batch.add(U, fixed_params(1, limiter=_capi.MC), (0, 0), fixed_steps=True)
        assert batch.status(sid)[0].c_h == r.c_h
    finally:
        batch.close()
    assert np.isfinite(r.c_h) and r.steps == 1
    if not infinite:
        want = signal_speed(U)
        assert abs(r.c_h - want) <= 2e-6 * want

"""The device generator of Fourier states at the edges of its work split (256 cells of a row per item,
kx and ky in chunks of 32; spectra and partials in the free scratch planes or, on tiny grids, in
buffers of their own) against the host generator. Both evaluate the same sums in FP64 in different
orders: kmax^2 terms of magnitude <= 1 give at most a few 1e-14 relative; held to 1e-12."""

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (31, 40), (255, 9), (256, 8), (257, 33)])
@pytest.mark.parametrize("kmax", [1, 8, 31, 33])
def test_fourier_generator_matches_host(nx, ny, kmax):
    want = wl.to_conservative(wl.fourier_state(nx, ny, 4, kmax), 5.0 / 3.0)
    dev = _capi.DeviceSolver(nx, ny)
    try:
        dev.configure(_capi.BC_PERIODIC, _capi.BC_PERIODIC)
        dev.generate(_capi.InitSpec.fourier(4, kmax), _capi.make_params())
        got = dev.download()[:, 2:-2, 2:-2]
    finally:
        dev.close()
    scale = np.abs(want).reshape(9, -1).max(axis=1)
    err = np.abs(got - want).reshape(9, -1).max(axis=1)
    assert np.all(err <= 1e-12 * np.maximum(1.0, scale)), err

"""FP64 states far from one. A speed that overflows has to end a solve by its time step, as in the
reference, through every FP64 entry point; states in units of density and velocity that take
gamma p + B^2 to 2^532 (its square overflows, squares of momenta do not) or to 2^-500, and states with
cells without pressure, have to follow the oracle. Held to the FP64 bar of the other parity tests
(relative L1 1e-12 per component): units that are powers of two change no rounding."""

import ctypes as C

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200 import workloads as wl
from mhd_gpu_solver_b200.batch import BatchSolver, fixed_params
from oracle import oracle as orc
from tests.gpu_util import gpu_solve
from tests.helpers import initial_state

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0


def _no_alloc(U, params, nsteps):
    import torch

    ny, nx = U.shape[1] - 4, U.shape[2] - 4
    u_in = torch.from_numpy(np.ascontiguousarray(U[:, 2:-2, 2:-2])).cuda()
    u_out = torch.empty_like(u_in)
    torch.cuda.synchronize()
    g, r = _capi.Grid(nx, ny, 2, 0.0, 1.0, 0.0, 1.0), _capi.Result()
    rc = _capi.lib.mhdb_solve_steps_noalloc_f64(
        C.byref(g), 0, 0, C.byref(params), nsteps, C.c_void_p(u_in.data_ptr()),
        C.c_void_p(u_out.data_ptr()), C.byref(r), None)
    return rc, u_out.cpu().numpy()


@pytest.mark.parametrize("nx,ny", [(45, 37), (500, 470)])
def test_speed_that_overflows_ends_the_solve(nx, ny):
    prim = wl.fourier_state(nx, ny, 4)
    prim["p"][ny // 2, nx // 3] = 1e160
    U0 = initial_state(prim, GAMMA)
    dev = _capi.DeviceSolver(nx, ny)
    try:
        for config in [-1] + [c["config"] for c in _capi.tile_configs(_capi.FP64)]:
            dev.set_tile_config(config)
            dev.configure(_capi.BC_PERIODIC, _capi.BC_PERIODIC)
            dev.upload(U0)
            with pytest.raises((ValueError, RuntimeError), match="positive dt"):
                dev.solve_steps(_capi.make_params(limiter=_capi.MC), 3)
    finally:
        dev.close()
    batch = BatchSolver(_capi.FP64)
    try:
        sid = batch.add(U0, fixed_params(3, limiter=_capi.MC), (0, 0), fixed_steps=True)
        batch.step(3)
        with pytest.raises((ValueError, RuntimeError), match="positive dt"):
            batch.status(sid)
    finally:
        batch.close()
    if nx < 100:  # the larger grid is beyond the allocation-free solve's scratch
        rc, _ = _no_alloc(U0, _capi.make_params(limiter=_capi.MC), 3)
        assert rc == _capi.BAD_TIMESTEP


def _l1(a, b):
    a, b = (x.reshape(9, -1) for x in (a, b))
    top = np.abs(b).max(axis=1, keepdims=True)
    top[top == 0.0] = 1.0
    return (np.abs(a - b) / top).sum(axis=1) / np.maximum((np.abs(b) / top).sum(axis=1), 1.0)


def _state(kind, nx, ny):
    prim = wl.fourier_state(nx, ny, 5)
    if kind == "no_pressure":  # at rest and without field, so that the energy is zero exactly
        block = (slice(ny // 4, ny // 2), slice(nx // 4, nx // 2))
        for k in ("p", "vx", "vy", "vz", "bx", "by", "bz"):
            prim[k][block] = 0.0
    U0 = initial_state(prim, GAMMA)
    if kind != "no_pressure":
        rho, v = (2.0 ** 332, 2.0 ** 100) if kind == "large" else (2.0 ** -460, 2.0 ** -20)
        U0[0] *= rho
        U0[1:4] *= rho * v
        U0[4] *= rho * v * v
        U0[5:8] *= np.sqrt(rho) * v
    return U0


@pytest.mark.parametrize("limiter", [orc.MINMOD, orc.MC, orc.VANLEER])
@pytest.mark.parametrize("kind", ["large", "small", "no_pressure"])
def test_far_units_and_empty_cells_match_oracle(kind, limiter):
    nx, ny = 61, 45
    U0 = _state(kind, nx, ny)
    p = orc.Params(limiter=limiter, max_steps=4, fixed_steps=True)
    ref, t, steps, c_h = orc.solve(U0, orc.Grid(nx, ny), p)
    assert np.isfinite(ref).all()
    want = ref[:, 2:-2, 2:-2]
    for config in [-1] + [c["config"] for c in _capi.tile_configs(_capi.FP64)]:
        got, tg, sg, cg = gpu_solve(U0, orc.Grid(nx, ny), p, tile_config=config)
        assert sg == steps and abs(tg - t) <= 1e-12 * t and abs(cg - c_h) <= 1e-12 * c_h
        err = _l1(got[:, 2:-2, 2:-2], want)
        assert np.all(err <= 1e-12), (config, err)
    rc, got = _no_alloc(U0, _capi.make_params(limiter=limiter), 4)
    assert rc == _capi.OK and np.all(_l1(got, want) <= 1e-12)

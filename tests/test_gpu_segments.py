"""The stage launches of a solve are replayed as graphs; with event profiling on they are launched
one by one. Both must give the same bits, on grids of one partial wave of blocks, about one wave
and many, in every default form. Strip marches cut a grid into segments by its size
(segment_rows): the result must match the oracle whatever the cut, ragged last segments of one
row and grids smaller than a strip included."""

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200 import workloads as wl
from oracle import oracle as orc
from tests.gpu_util import gpu_solve
from tests.helpers import assert_components, initial_state

pytestmark = pytest.mark.gpu

NONIDEAL = dict(ohmic=True, hall=True, ambipolar=True, eta_ohm=1e-3, eta_hall=1e-2,
                eta_ambipolar=1e-3)


@pytest.mark.parametrize("precision", [_capi.FP64, _capi.FP32])
@pytest.mark.parametrize("nx,ny,nonideal", [(96, 80, False), (520, 300, True), (1024, 1024, False),
                                            (2048, 2048, False)])
def test_graph_launches_give_the_bits_of_single_ones(precision, nx, ny, nonideal):
    params = _capi.make_params(limiter=_capi.VANLEER, **(NONIDEAL if nonideal else {}))
    init = _capi.InitSpec.fourier(5)
    outs = []
    for plain in (True, False, False):
        dev = _capi.DeviceSolver(nx, ny, precision=precision)
        try:
            dev.configure(_capi.BC_PERIODIC, _capi.BC_OUTFLOW)
            dev.generate(init, params)
            dev.set_profiling(plain)
            r = dev.solve_steps(params, 45)  # one graph of 32 steps and 13 direct ones
            outs.append((dev.download(), r.t, r.steps, r.c_h))
        finally:
            dev.close()
    for got in outs[1:]:
        assert got[1:] == outs[0][1:]
        assert np.array_equal(got[0], outs[0][0])


@pytest.mark.parametrize("nx,ny", [(1, 1), (29, 2), (57, 33), (61, 70), (300, 65)])
@pytest.mark.parametrize("precision,config,tol", [(_capi.FP64, 7, 1e-12), (_capi.FP64, 8, 1e-12),
                                                  (_capi.FP32, 17, 1e-6), (_capi.FP32, 18, 1e-6)])
def test_segments_cut_to_the_grid_match_oracle(precision, config, tol, nx, ny):
    U0 = initial_state(wl.fourier_state(nx, ny, 2), 5.0 / 3.0, (orc.OUTFLOW, orc.PERIODIC))
    p = orc.Params(limiter=orc.VANLEER, max_steps=6, fixed_steps=True, **NONIDEAL)
    ref, t, steps, c_h = orc.solve(U0, orc.Grid(nx, ny), p, (orc.OUTFLOW, orc.PERIODIC))
    got, tg, sg, _ = gpu_solve(U0, orc.Grid(nx, ny), p, (orc.OUTFLOW, orc.PERIODIC),
                               precision=precision, tile_config=config)
    assert sg == steps and abs(tg - t) <= 1e-6 * t
    assert_components(got, ref, tol, c_h)

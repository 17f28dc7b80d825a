"""The strip marches' row loop on small grids. By default a small grid is cut into segments of one row,
which leaves out all that a march carries from row to row (primitives, slopes, fluxes and currents,
the halo ring's slots and phases, the increment ring, mask bytes). Here the segments' height is set:
one row, fewer rows than the rings hold, just more, and the whole tile, each with a ragged last
segment, against the FP64 oracle at the bars of the other parity tests (relative L1 1e-12 for FP64,
1e-6 for FP32-mixed)."""

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200 import workloads as wl
from oracle import oracle as orc
from tests.gpu_util import to_c_params
from tests.helpers import assert_components, initial_state

pytestmark = pytest.mark.gpu

NONIDEAL = dict(ohmic=True, hall=True, ambipolar=True, eta_ohm=1e-3, eta_hall=1e-2,
                eta_ambipolar=1e-3)
NX, NY, STEPS = 61, 71, 7
ROWS = [2, 3, 5, 32, 64]  # 71 rows leave 1, 2, 1, 7 and 7 for the last segment
TOL = {_capi.FP64: 1e-12, _capi.FP32: 1e-6}


def _marches(precision):
    return [c for c in _capi.tile_configs(precision)
            if c["kind"].startswith("march") and c["kind"] != "march_tma_pair"]


def _mask():
    """Solid cells on the edges and inside, isolated ones and blocks among them."""
    rng = np.random.Generator(np.random.PCG64(17))
    mask = (rng.uniform(size=(NY, NX)) > 0.06).astype(np.uint8)
    mask[20:31, 24:37] = 0
    mask[0, 5:9] = mask[-1, 40:47] = mask[33:40, 0] = mask[50:54, -1] = 0
    return mask


def _run(U0, p, bc, precision, config, rows, mask=None, walls=True):
    dev = _capi.DeviceSolver(NX, NY, precision=precision)
    try:
        dev.set_tile_config(config)
        dev.debug_segment_rows(rows)
        dev.configure(bc[0], bc[1], mask, walls)
        dev.upload(U0)
        r = dev.solve_steps(to_c_params(p), p.max_steps)
        return dev.download(), r
    finally:
        dev.close()


@pytest.mark.parametrize("precision", [_capi.FP64, _capi.FP32])
@pytest.mark.parametrize("limiter,bc,nonideal", [
    (orc.VANLEER, (orc.PERIODIC, orc.OUTFLOW), False), (orc.MC, (orc.OUTFLOW, orc.PERIODIC), True),
    (orc.MINMOD, (orc.PERIODIC, orc.PERIODIC), False), (orc.VANLEER, (orc.OUTFLOW, orc.OUTFLOW), True)])
def test_segments_of_several_rows_match_oracle(precision, limiter, bc, nonideal):
    U0 = initial_state(wl.fourier_state(NX, NY, 7), 5.0 / 3.0, bc)
    p = orc.Params(limiter=limiter, max_steps=STEPS, fixed_steps=True,
                   **(NONIDEAL if nonideal else {}))
    ref, t, steps, c_h = orc.solve(U0, orc.Grid(NX, NY), p, bc)
    for cfg in _marches(precision):
        for rows in ROWS:
            got, r = _run(U0, p, bc, precision, cfg["config"], rows)
            assert r.steps == steps and abs(r.t - t) <= TOL[precision] * t
            assert_components(got, ref, TOL[precision], c_h, what=(cfg, rows))


@pytest.mark.parametrize("precision,configs", [(_capi.FP64, [7]), (_capi.FP32, [11, 13, 17])])
@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("nonideal", [False, True])
def test_masked_segments_of_several_rows_match_oracle(precision, configs, walls, nonideal):
    bc = (orc.OUTFLOW, orc.PERIODIC)
    mask = _mask()
    U0 = initial_state(wl.fourier_state(NX, NY, 6), 5.0 / 3.0, bc, mask, walls)
    p = orc.Params(limiter=orc.VANLEER, max_steps=STEPS, fixed_steps=True,
                   **(NONIDEAL if nonideal else {}))
    ref, t, steps, c_h = orc.solve(U0, orc.Grid(NX, NY), p, bc, mask, walls)
    for config in configs:
        for rows in ROWS:
            got, r = _run(U0, p, bc, precision, config, rows, mask, walls)
            assert r.steps == steps and abs(r.t - t) <= TOL[precision] * t
            assert_components(got, ref, TOL[precision], c_h, what=(config, rows))


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("rows", ROWS)
def test_increment_ring_gives_the_bits_of_the_own_stream(rows, masked):
    """Configuration 17 takes the own cells' increment from a three-row ring, configuration 13 from a
    stream of its own: the same operands, so the same bits, whatever the segments' height."""
    bc = (orc.PERIODIC, orc.OUTFLOW)
    mask = _mask() if masked else None
    U0 = initial_state(wl.fourier_state(NX, NY, 8), 5.0 / 3.0, bc, mask)
    p = orc.Params(limiter=orc.VANLEER, max_steps=STEPS, fixed_steps=True)
    (a, ra), (b, rb) = (_run(U0, p, bc, _capi.FP32, c, rows, mask) for c in (13, 17))
    assert ra.t == rb.t and np.array_equal(a, b)


def test_height_beyond_the_tallest_tile_is_refused():
    dev = _capi.DeviceSolver(NX, NY)
    try:
        for rows in (-1, 65):
            with pytest.raises(ValueError):
                dev.debug_segment_rows(rows)
    finally:
        dev.close()

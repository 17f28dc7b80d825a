"""The FP64 kernels' own reciprocal, roots and fallback test against the CPU oracle, on states that
reach their edges: no field at all (the inner root of the fast speed is gamma p exactly), field
along one axis with gamma p = B^2 (its argument is zero or a rounding error of either sign), cold
cells, and contrasts that make second-order face states negative, so that whole faces fall back to
first order. Held to the FP64 bar (relative L1 1e-12 per component: a few roundings of 1e-16 in
each of some hundred operations of a face, a few steps), on the tile kernel and the strip march."""

import numpy as np
import pytest

from mhd_gpu_solver_b200 import workloads as wl
from oracle import oracle as orc
from tests.gpu_util import gpu_solve
from tests.helpers import assert_components, initial_state

pytestmark = pytest.mark.gpu

NX, NY, GAMMA = 45, 37, 5.0 / 3.0


def _state(kind):
    s = wl.fourier_state(NX, NY, 3)
    rng = np.random.Generator(np.random.PCG64(11))
    if kind == "no_field":
        s["bx"][:] = s["by"][:] = 0.0
    elif kind in ("aligned_x", "aligned_y"):
        along, across = ("bx", "by") if kind == "aligned_x" else ("by", "bx")
        s[across][:] = 0.0
        s[along] = np.sqrt(GAMMA * s["p"])
    elif kind == "cold":
        s["p"][:] = 1e-4
        s["p"][::3, ::4] = 1e-6
        s["vx"] *= 1e-2
        s["vy"] *= 1e-2
    else:  # contrasts
        s["rho"] = 10.0 ** rng.uniform(-3.0, 0.0, size=(NY, NX))
        s["p"] = 10.0 ** rng.uniform(-3.0, 0.0, size=(NY, NX))
        s["bx"] *= 0.05
        s["by"] *= 0.05
        s["vx"] *= 0.05
        s["vy"] *= 0.05
    return s


@pytest.mark.parametrize("config", [2, 7])
@pytest.mark.parametrize("limiter", [orc.MINMOD, orc.MC, orc.VANLEER])
@pytest.mark.parametrize("kind", ["no_field", "aligned_x", "aligned_y", "cold", "contrasts"])
def test_f64_kernels_at_the_edges_of_their_arithmetic(kind, limiter, config):
    U0 = initial_state(_state(kind), GAMMA)
    p = orc.Params(limiter=limiter, max_steps=3, fixed_steps=True)
    ref, t, steps, c_h = orc.solve(U0, orc.Grid(NX, NY), p)
    got, tg, sg, cg = gpu_solve(U0, orc.Grid(NX, NY), p, tile_config=config)
    assert sg == steps and abs(tg - t) <= 1e-12 * t and abs(cg - c_h) <= 1e-12 * c_h
    assert_components(got, ref, 1e-12, c_h, what=(kind, limiter, config))

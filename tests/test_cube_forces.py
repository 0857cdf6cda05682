"""DFSPH in a cube boundary with force plugins.

The cube clamps positions after the grid build (DFSPHSolver::step), so the next step's forces see other distances
than the build did: pairs that the clamp brings together must take part.  One scene with its solver's iterations
switched off, thrown at the walls fast enough to be clamped every step by a part of the support radius, with lists
and with cell walks (neighbor_list_max = 0), at a size whose list build has several lanes per particle and at one
whose build has one."""
import numpy as np
import pytest

import sph_gb300
from scenes import lattice

pytestmark = pytest.mark.gpu

R = 0.02
STEPS = 4


def thrown(side, precision, lists, lanes):
    d = 2 * R
    x = lattice(R, (0, 0, 0), (d * side + 1e-9,) * 3)
    assert len(x) == side**3
    rng = np.random.default_rng(side)
    x = x + rng.uniform(-0.3 * R, 0.3 * R, x.shape)
    v = rng.uniform(-1, 1, x.shape)
    v[:, 0] -= 5.0
    p = dict(method=2, boundary=0, has_cube=1, cube_min=(0.0, 0.0, 0.0), cube_max=(d * side + 8 * R,) * 3, radius=R,
             dt=2e-3, min_dt=2e-3, max_dt=2e-3, min_it=0, max_it=0, min_it_v=0, max_it_v=0, visc_method=2, visc=0.5)
    if precision == "f64":
        p.update(st_method=3, st=0.5)
    s = sph_gb300.Scene(precision=precision, neighbor_list_max=lists, threads_per_particle=lanes, **p)
    s.set_fluid(x, v)
    s.init()
    s.step(STEPS)
    return s.get("v")


@pytest.mark.parametrize("side,lanes", [(9, 8), (9, 1), (30, 1), (30, 4)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_forces_see_clamped_positions(gpu_lib, precision, side, lanes):
    a, w = (thrown(side, precision, n, lanes) for n in (64, 0))
    # the densities of the two builds differ by their rounding (64 terms), the forces by theirs; each step adds at
    # most 0.5 * 64 * |v_j - v_i| W m / rho (XSPH), and in FP64 the surface tension's terms of the same order
    eps = 2.0**-24 if precision == "f32" else 2.0**-53
    assert np.abs(a - w).max() <= STEPS * 2 * 64 * eps * np.abs(w).max()

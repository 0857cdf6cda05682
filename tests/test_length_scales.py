"""Neighbour lists of scenes of any length unit.

The list builds cull candidates from half-precision positions.  Half precision has 5 exponent bits: the same scene
must keep every neighbour from a radius of a tenth of a millimetre (squares of the distances below its normal range)
to one of kilometres (distances above its largest value)."""
import numpy as np
import pytest

import sph_gb300
from scenes import lattice

pytestmark = pytest.mark.gpu

RADII = [1e-12, 7.3e-5, 9.4e-5, 1.5e-4, 0.01, 3e4, 1e9]


def block(r, side=9):
    x = lattice(1.0, (4, 4, 4), (4 + 2 * side + 1e-6,) * 3)
    x = (x + np.random.default_rng(11).uniform(-0.3, 0.3, x.shape)) * r
    b = sph_gb300.sample_box(4.0, (0, 0, 0), (2 * side + 8,) * 3) * r
    return x, b


def scene(r, lists, precision, lanes, **p):
    x, b = block(r)
    s = sph_gb300.Scene(radius=r, boundary=2, precision=precision, neighbor_list_max=lists, threads_per_particle=lanes,
                        gravity=(0.0, 0.0, 0.0), **p)
    s.set_fluid(x)
    s.add_boundary_points(b)
    s.init()
    return s


@pytest.mark.parametrize("r", RADII)
@pytest.mark.parametrize("method", ["dfsph", "wcsph", "pcisph"])
@pytest.mark.parametrize("precision,lanes", [("f64", 1), ("f64", 8), ("f32", 1), ("f32", 8)])
def test_densities_with_lists_are_those_of_cell_walks(gpu_lib, r, method, precision, lanes):
    if precision == "f32" and not 1e-5 < r < 1e5:
        pytest.skip("kernel constants of order 1 / h^9 leave FP32")
    p = {"dfsph": dict(method=2), "wcsph": dict(method=0, dt=1e-12), "pcisph": dict(method=1, dt=1e-12, min_it=0, max_it=0)}[method]
    out = []
    for lists in (64, 0):
        s = scene(r, lists, precision, lanes, **p)
        if method != "dfsph":  # (DFSPH's are formed by init)
            s.step(1)
        out.append(s.get("rho"))
    # sums of at most 64 terms, in another order or with another rounding of the kernel's terms
    eps = 2.0**-24 if precision == "f32" else 2.0**-53
    assert np.abs(out[0] - out[1]).max() <= 2 * 64 * eps * np.abs(out[1]).max()


def check_neighbours(x, h, lists):
    """Every pair well inside the support is listed, none well outside (1e-4 h either side: positions in FP32)."""
    d = np.sqrt(((x[:, None, :] - x[None, :, :]) ** 2).sum(2))
    np.fill_diagonal(d, np.inf)
    listed = np.zeros(d.shape, bool)
    listed[np.repeat(np.arange(len(x)), np.diff(lists["off"])), lists["nbr"]] = True
    assert np.array_equal(np.diff(lists["off"]), lists["count"])
    assert not (~listed & (d < h * (1 - 1e-4))).any()
    assert not (listed & (d > h * (1 + 1e-4))).any()


@pytest.mark.parametrize("r", [r for r in RADII if 1e-5 < r < 1e5])
@pytest.mark.parametrize("where", ["scene", "scene_f64", "pool"])
def test_stored_neighbours(gpu_lib, r, where):
    x, b = block(r)
    p = dict(method=2, boundary=2, radius=r, gravity=(0.0, 0.0, 0.0), dt=1e-12, min_dt=1e-12, max_dt=1e-12, min_it=0, max_it=0,
             min_it_v=0, max_it_v=0)
    if where != "pool":
        s = sph_gb300.Scene(neighbor_list_max=64, precision="f64" if where == "scene_f64" else "f32", **p)
        s.set_fluid(x)
        s.add_boundary_points(b)
        s.init()
        check_neighbours(s.get("x"), 4 * r, s.pair_lists())
        return
    # beside a scene of another scale
    P = sph_gb300.Pool(max_particles=2 * len(x), max_boundary=2 * len(b), max_keys=200_000, max_scenes=2)
    P.set_autotune(0)
    x2, b2 = block(0.02)
    ids = [P.add_scene(x, boundary_points=b, steps=2, precision="f32", **p),
           P.add_scene(x2, boundary_points=b2, steps=2, precision="f32", **dict(p, radius=0.02))]
    P.step(1)
    for k, rr in zip(ids, (r, 0.02)):
        check_neighbours(P.get(k, "x"), 4 * rr, P.pair_lists(k))

"""Force passes over candidate lists against cell walks (neighbor_list_max = 0).

* PCISPH with several lanes per particle: velocities and pressure accelerations of a compressed block.
* WCSPH with XSPH: the one pass of both forces against the two walks.
* DFSPH with every force plugin at sizes whose list build has one lane per particle and writes the candidate lists
  itself, with 1 to 8 lanes in the force passes, with lists that hold every candidate and lists that do not.
* DFSPH scenes of several lanes per particle with lists on either side of the length from which they are built so: the
  solver's first divergence error, formed by the build or by a pass of its own.
* Every set of force plugins: FP32 compiles most of them apart over lists, whose sums stay the walk's.
* A WCSPH step's phases with lists."""
import numpy as np
import pytest

import sph_gb300
from scenes import lattice

pytestmark = pytest.mark.gpu

R = 0.02
FORCES = dict(visc_method=2, visc=0.01, bvisc=0.01, st_method=3, st=0.5, adh_method=4, adh=0.1)
EPS = {"f32": 2.0**-24, "f64": 2.0**-53}


def block(n, spacing=1.0, seed=5):
    side = int(np.ceil(n ** (1 / 3)))
    x = lattice(R, (2 * R,) * 3, (2 * R + 2 * R * side + 1e-9,) * 3)[:n]
    x = x * spacing + np.random.default_rng(seed).uniform(-0.1 * R, 0.1 * R, x.shape)
    return x, np.random.default_rng(seed + 1).uniform(-0.2, 0.2, x.shape)


def run(x, v, fields, steps=1, **p):
    e = float(x.max()) + 4 * R
    s = sph_gb300.Scene(boundary=2, radius=R, **p)
    s.set_fluid(x, v)
    s.add_boundary_points(sph_gb300.sample_box(4 * R, (0, 0, 0), (e, e, e)))
    s.init()
    s.step(steps)
    return [s.get(f) for f in fields]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("lanes,lists", [(8, 64), (4, 64), (2, 64), (8, 40), (8, 30), (8, 1), (4, 40), (2, 42)])
@pytest.mark.parametrize("n", [17, 600])
def test_pcisph_lanes(gpu_lib, precision, lanes, lists, n):
    x, v = block(n, 0.85)
    p = dict(method=1, precision=precision, threads_per_particle=lanes, dt=1e-4, min_it=2, max_it=2, eta=0.001, **FORCES)
    a, w = (run(x, v, ("v", "pacc"), neighbor_list_max=k, **p) for k in (lists, 0))
    if n == 600:
        assert np.abs(w[1]).max() > 1.0  # compressed: pressures act
    for g, e in zip(a, w):
        if precision == "f32":
            # each lane's list is its share of the walk, in its order
            assert np.array_equal(g, e)
        else:
            # 64 terms in another order; a pressure from a density error of at least 1 % of the density
            assert np.abs(g - e).max() <= 64 * 64 * EPS["f64"] / 0.01 * np.abs(e).max()


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n", [127, 129, 1500])
def test_wcsph_forces_of_one_pass(gpu_lib, precision, n):
    x, v = block(n, 0.95)
    p = dict(method=0, precision=precision, threads_per_particle=1, dt=1e-4, visc_method=2, visc=0.05, bvisc=0.02)
    (a,), (w,) = (run(x, v, ("v",), neighbor_list_max=k, steps=1 if precision == "f32" else 10, **p) for k in (64, 0))
    if precision == "f64":
        # one lane: the walk's terms in the walk's order, and quotients that round as divisions
        assert np.array_equal(a, w)
    else:
        # 64 terms of p / rho^2 m |grad W| dt, p = k ((rho / rho0)^7 - 1) with k = 1.43e5 and (rho / rho0)^7 <= 4
        assert np.abs(a - w).max() <= 64 * EPS["f32"] * 64 * 2 * 3 * 1.43e5 / 1e6 * 500 * 1e-4


VISCOSITY = {"none": {}, "xsph": dict(visc_method=2, visc=0.01, bvisc=0.01), "standard": dict(visc_method=0, visc=0.01, bvisc=0.01),
             "artificial": dict(visc_method=1, visc=0.01, bvisc=0.01)}


@pytest.mark.parametrize("precision,lanes", [("f32", 1), ("f32", 4), ("f64", 1)])
@pytest.mark.parametrize("visc", list(VISCOSITY))
@pytest.mark.parametrize("tension", [0, 1])
@pytest.mark.parametrize("adhesion", [0, 1])
def test_force_sets(gpu_lib, precision, lanes, visc, tension, adhesion):
    if visc == "none" and not tension and not adhesion:
        pytest.skip("no plugin")
    x, v = block(500)
    p = dict(method=1, precision=precision, threads_per_particle=lanes, dt=1e-4, min_it=2, max_it=2, eta=0.001, **VISCOSITY[visc])
    if tension:
        p.update(st_method=3, st=0.5)
    if adhesion:
        p.update(adh_method=4, adh=0.1)
    a, w = (run(x, v, ("v", "x"), steps=2, neighbor_list_max=k, **p) for k in (64, 0))
    for g, e in zip(a, w):
        assert np.array_equal(g, e)


def sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("lists", [64, 33, 30])
@pytest.mark.parametrize("where", ["one", "one_eight_blocks"])
def test_dfsph_forces_over_lists_of_the_build(gpu_lib, precision, lanes, lists, where):
    """One particle more than the sizes with several lanes per particle in the build, and (FP64) than those with six
    resident blocks per SM."""
    if where == "one_eight_blocks" and (precision == "f32" or lanes in (2, 4)):
        pytest.skip("FP64 only; 1 and 8 lanes")
    n = sms() * (5 * 32 if where == "one" else 6 * 128) + 1
    x, v = block(n)
    p = dict(method=2, precision=precision, threads_per_particle=lanes, dt=1e-3, min_dt=1e-3, max_dt=1e-3, min_it=0, max_it=0,
             min_it_v=0, max_it_v=0, **FORCES)
    (a,), (w,) = (run(x, v, ("v",), neighbor_list_max=k, **p) for k in (lists, 0))
    # the builds' densities differ by 64 roundings, a force term by as many; 64 terms of at most 10 m/s^2 a particle
    assert np.abs(a - w).max() <= 4 * 64 * EPS[precision] * (np.abs(w).max() + 64 * 10 * 1e-3)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n", [600, 30000])  # 8 lanes and one lane per particle in the build
def test_short_lists(gpu_lib, precision, n):
    x, v = block(n, 0.98)
    p = dict(method=2, precision=precision, threads_per_particle=4, dt=1e-4, min_dt=1e-4, max_dt=1e-4, min_it=0, max_it=0, min_it_v=1,
             max_it_v=1, visc_method=2, visc=0.05)
    out = [run(x, v, ("rho", "div", "v"), neighbor_list_max=k, **p) for k in (31, 32, 64)]
    eps = EPS[precision]
    for rho, div, vel in out[:2]:
        r0, d0, v0 = out[2]
        # overflowed particles walk the cells, whose kernel values round otherwise: 64 terms; a divergence of 64 terms of
        # at most 0.7 m/s * 500 / (m s)
        assert np.abs(rho - r0).max() <= 2 * 64 * eps * np.abs(r0).max()
        close = np.abs(div - d0) <= 4 * 64 * eps * 64 * 0.7 * 500
        # (a pair at the support to rounding decides the rule of 20 neighbours: a free surface has a few such particles)
        assert close.mean() >= (1.0 if precision == "f64" else 0.999)
        assert np.median(np.abs(vel - v0)) <= 64 * eps * np.abs(v0).max()


def test_wcsph_phases_with_lists(gpu_lib):
    """Pressure force and viscosity of one pass are timed under both names, joined."""
    x, v = block(600)
    s = sph_gb300.Scene(method=0, boundary=2, radius=R, precision="f32", visc_method=2, visc=0.01, dt=1e-4, neighbor_list_max=64)
    s.set_fluid(x, v)
    s.add_boundary_points(sph_gb300.sample_box(4 * R, (0, 0, 0), (0.6, 0.6, 0.6)))
    s.init()
    s.set_profiling(True)
    s.step(3)
    ph = s.phase_profile()
    assert {k: n for k, (n, _) in ph.items()} == {"Step computation": 3, "Fill grid": 3, "Densities+Pressures": 3,
                                                  "Pressure force+NPForces": 3, "Integratio": 3}

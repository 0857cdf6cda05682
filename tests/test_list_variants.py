"""Variants of the neighbour-list passes at the sizes where their branches part.

* Candidate lists whose fluid candidates fit but whose boundary candidates do not (those are then walked): the
  passes must still give the cell walks' results bit for bit.
* The DFSPH list build that also forms the divergence solve's first error pass, at block edges.
* The list build with 8, 4 and 1 lanes per particle (chosen by scene size), with lists that hold every neighbour and
  lists that overflow.
* Candidate lists built and visited by several lanes per particle.
* Particles whose candidates overflow the build's queue but whose neighbours fit the list.
* The FP64 list build with eight blocks per SM, on either side of the size that chooses it.
* The grid's key scan in two launches and in three, at the edges of its tiles.
"""
import numpy as np
import pytest

import sph_gb300
from scenes import jitter, lattice
from test_pcisph_lists import drop, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,precision,lists", [("impact", "f32", 44), ("impact", "f64", 40), ("wcsph", "f32", 34)])
def test_boundary_candidates_beyond_the_list(gpu_lib, case, precision, lists):
    x, v, b, p = drop(case)
    a, w = (run(x, v, b, p, precision, n, 12, True) for n in (lists, 0))
    for f in ("x", "v", "rho"):
        assert np.array_equal(a.get(f), w.get(f)), f


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n", [127, 128, 129, 700])
def test_first_divergence_error_formed_by_the_build(gpu_lib, precision, n):
    """The list build's half-precision cull and the divergence error it forms, over one block, one particle less or
    more, and a part of a block: FP64 against walks of every cell (neighbor_list_max = 0), FP32 against the same scene
    in a pool (a walk's kernel values round differently there, and a pair at the support radius may count for one
    of them and not for the other, which decides the solver's rule of 20 neighbours)."""
    r = 0.02
    x = jitter(lattice(r, (2 * r, 2 * r, 2 * r), (0.45, 0.45, 0.45)), r, 3)[:n]
    v = np.random.default_rng(n).uniform(-0.2, 0.2, x.shape)
    p = dict(method=2, boundary=2, radius=r, precision=precision, eta=0.001, eta_v=0.001, max_it_v=0, min_it_v=0)
    b = sph_gb300.sample_box(4 * r, (0, 0, 0), (0.6, 0.6, 0.6))

    def alone(lists):
        s = sph_gb300.Scene(neighbor_list_max=lists, threads_per_particle=1, **p)
        s.set_fluid(x, v)
        s.add_boundary_points(b)
        s.init()
        s.step(1)
        return s.get("rho"), s.get("alpha"), s.get("div"), s.stats()["iterations"]

    def pooled():
        P = sph_gb300.Pool(max_particles=n, max_boundary=len(b), max_keys=100_000, max_scenes=2)
        P.set_autotune(0)
        k = P.add_scene(x, v=v, boundary_points=b, steps=2, **p)
        P.step(1)
        return P.get(k, "rho"), P.get(k, "alpha"), P.get(k, "div"), P.query(k)[0]["iterations"]

    rho, alpha, div, it = alone(64)
    rho0, alpha0, div0, it0 = pooled() if precision == "f32" else alone(0)
    # sums of up to ~60 terms, the boundary's pre-added in the lists: 60 roundings of the largest value
    tol = 60 * (2.0**-24 if precision == "f32" else 2.0**-53)
    assert it == it0
    for a, e, scale in ((rho, rho0, 1.0), (alpha, alpha0, 4.0)):
        assert np.abs(a - e).max() <= scale * tol * np.abs(e).max()
    # a divergence sums terms of either sign: bound by the sum of their sizes, |v_i - v_j| |m grad W| <= 0.7 * 60 * 500
    assert np.abs(div - div0).max() <= tol * 0.7 * 60 * 500


@pytest.mark.parametrize("lists", [64, 24])
@pytest.mark.parametrize("side", [(1, 1, 1), (5, 3, 3), (21, 21, 22), (22, 21, 21), (23, 23, 23), (29, 29, 29), (30, 29, 29)])
def test_build_lanes_match_the_pool(gpu_lib, side, lists):
    """One scene (lanes by size: the sides around 9.7k and 24k particles change them) against the same scene in a pool
    (one lane): the same neighbours in the same order, the same sums up to their rounding."""
    r = 0.01
    d = 2 * r
    x = lattice(r, (d, d, d), tuple(d + d * k + 1e-9 for k in side))
    assert x.shape[0] == side[0] * side[1] * side[2]
    rng = np.random.default_rng(7)
    # jittered enough that no pair lies at the support radius to rounding
    x = x + rng.uniform(-0.2 * r, 0.2 * r, x.shape)
    v = rng.uniform(-0.2, 0.2, x.shape)
    p = dict(method=2, boundary=2, radius=r, precision="f32", eta=0.001, eta_v=0.001)
    b = sph_gb300.sample_box(4 * r, (0, 0, 0), (0.8, 0.8, 0.8))
    s = sph_gb300.Scene(neighbor_list_max=lists, **p)
    s.set_fluid(x, v)
    s.add_boundary_points(b)
    s.init()
    s.step(1)
    P = sph_gb300.Pool(max_particles=len(x), max_boundary=len(b), max_keys=200_000, max_scenes=2, neighbor_list_max=lists)
    P.set_autotune(0)
    k = P.add_scene(x, v=v, boundary_points=b, steps=2, **p)
    P.step(1)
    a, e = s.pair_lists(), P.pair_lists(k)
    for f in ("count", "off", "nbr"):
        assert np.array_equal(a[f], e[f]), f
    # the one-scene / pool bounds of the smoke test
    for f, tol in (("x", 1e-6), ("rho", 1e-5), ("alpha", 4e-5)):
        g, w = s.get(f), P.get(k, f)
        assert np.abs(g - w).max() <= tol * np.abs(w).max(), f


@pytest.mark.parametrize("method", ["wcsph", "pcisph"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("lanes,lists", [(8, 64), (4, 64), (2, 64), (8, 30), (8, 1), (4, 40)])
@pytest.mark.parametrize("n", [1, 17, 600])
def test_candidate_lists_shared_by_lanes(gpu_lib, method, precision, lanes, lists, n):
    """Candidate lists built and visited by several lanes per particle against the cell walks, after one step: sums
    of at most 64 terms, added in another order."""
    r = 0.02
    d = 2 * r
    x = jitter(lattice(r, (d, d, d), (0.45, 0.45, 0.45)), r, 3)
    x = x[np.random.default_rng(n).permutation(len(x))[:n]]
    p = dict(boundary=2, radius=r, precision=precision, dt=1e-4, visc_method=2, visc=0.01, bvisc=0.01)
    p.update(dict(method=0) if method == "wcsph" else dict(method=1, min_it=1, max_it=1, eta=0.001))
    out = []
    for k in (lists, 0):
        s = sph_gb300.Scene(threads_per_particle=lanes, neighbor_list_max=k, **p)
        s.set_fluid(x, np.random.default_rng(5).uniform(-0.2, 0.2, x.shape))
        s.add_boundary_points(sph_gb300.sample_box(4 * r, (0, 0, 0), (0.6, 0.6, 0.6)))
        s.init()
        s.step(1)
        out.append((s.get("rho"), s.get("v")))
    eps = 2.0**-24 if precision == "f32" else 2.0**-53
    (rho, v), (rho0, v0) = out
    assert np.abs(rho - rho0).max() <= 64 * eps * np.abs(rho0).max()
    if method == "wcsph":
        # p = k ((rho / rho0)^7 - 1), k = 1.43e5: 7 k 64 eps; 64 terms of 2 p / rho^2 times m |grad W| <= 500; dt
        assert np.abs(v - v0).max() <= 7 * 1.43e5 * 64 * eps * 2 / 1e6 * 64 * 500 * 1e-4


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("side", [7, 17, 31])  # 8, 4 lanes and 1 lane per particle
def test_lists_of_particles_whose_queue_overflows(gpu_lib, precision, side):
    """Slots for about the number of neighbours: more candidates than the queue holds, in particles whose lists still
    fit.  What is stored is what long lists hold, at the start and after a step's build."""
    r = 0.01
    e = 2 * r * (side + 1) + 1e-9
    x = jitter(lattice(r, (2 * r, 2 * r, 2 * r), (e, e, e)), r, 3)
    assert len(x) == side**3
    v = np.random.default_rng(side).uniform(-0.2, 0.2, x.shape)
    b = sph_gb300.sample_box(4 * r, (0, 0, 0), (e + 2 * r, e + 2 * r, e + 2 * r))

    def lists(kmax, steps):
        s = sph_gb300.Scene(neighbor_list_max=kmax, method=2, boundary=2, radius=r, precision=precision, max_it=0, min_it=0,
                            max_it_v=0, min_it_v=0)
        s.set_fluid(x, v)
        s.add_boundary_points(b)
        s.init()
        if steps:
            s.step(steps)
        return s.pair_lists()

    for steps in (0, 1):
        a, w = lists(30, steps), lists(64, steps)
        assert np.array_equal(a["count"], w["count"])
        fits = w["count"] <= 30
        assert fits.any() and not fits.all()
        assert np.array_equal(a["nbr"], w["nbr"][np.repeat(fits, w["count"])])


@pytest.mark.parametrize("lists", [64, 24])
def test_f64_build_by_size(gpu_lib, lists):
    """Five blocks of 128 particles per SM, and the same with one particle more that is far from all others: FP64 is
    compiled without contraction and the sums keep their order, so the two forms of the build agree bit for bit, with
    lists that hold every neighbour and with lists (and candidate queues) that overflow."""
    torch = pytest.importorskip("torch")
    n = torch.cuda.get_device_properties(0).multi_processor_count * 5 * 128
    r = 0.01
    side = int(np.ceil(n ** (1 / 3)))
    e = 2 * r * (side + 1) + 1e-9
    x = jitter(lattice(r, (2 * r, 2 * r, 2 * r), (e, e, e)), r, 3)[:n]
    v = np.random.default_rng(n).uniform(-0.2, 0.2, x.shape)
    b = sph_gb300.sample_box(4 * r, (0, 0, 0), (e + 2 * r, e + 2 * r, e + 2 * r))
    x = np.vstack([x, [[e + 20 * r, e, e]]])
    v = np.vstack([v, np.zeros((1, 3))])
    out = []
    for m in (n, n + 1):
        s = sph_gb300.Scene(neighbor_list_max=lists, method=2, boundary=2, radius=r, precision="f64", eta=0.001, eta_v=0.001,
                            max_it_v=0, min_it_v=0, domain_min=(-4 * r,) * 3, domain_max=(e + 30 * r,) * 3)
        s.set_fluid(x[:m], v[:m])
        s.add_boundary_points(b)
        s.init()
        s.step(1)
        out.append([s.get(f)[:n] for f in ("rho", "alpha", "div", "v")])
    for a, w in zip(*out):
        assert np.array_equal(a, w)


@pytest.mark.parametrize("cells", [(8, 5), (8, 32), (8, 33), (16, 40), (64, 512), (64, 513)])
def test_key_scan_tiles(gpu_lib, cells):
    """A part of a 2048-key tile, one tile, one and a part, five, 1024 (the last with the scan's sums folded into its
    second launch) and 1026, against the same particles in a box of 128 columns a side and at least 1100 tiles: the
    same neighbours, summed in another order (at most 60 terms)."""
    side, nz = cells
    r = 0.02
    h = 4 * r
    rng = np.random.default_rng(side * nz)
    top = (nz - 4) * h
    x = rng.uniform((0, 0, 0), (3 * h, 3 * h, min(top, 4 * h)), (60, 3))
    x[30:, 2] = top - x[30:, 2]  # at both ends of the keys
    x = np.clip(x, 1e-3 * h, (3.999 * h, 3.999 * h, top - 1e-3 * h))

    def density(s, z):
        lo = (0.5 * h, 0.5 * h, 0.5 * h)
        hi = ((s - 4.5) * h, (s - 4.5) * h, (z - 4.5) * h)
        sc = sph_gb300.Scene(method=0, boundary=2, radius=r, precision="f64", dt=1e-5, domain_min=lo, domain_max=hi)
        sc.set_fluid(x)
        sc.init()
        sc.step(1)
        return sc.get("rho")

    a, w = density(side, nz), density(128, max(nz, 138))
    assert np.abs(a - w).max() <= 60 * 2.0**-53 * np.abs(w).max()

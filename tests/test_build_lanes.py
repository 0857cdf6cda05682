"""The list build's forms by size (8, 4 and 1 lanes per particle, and in FP64 one lane with eight resident blocks per SM
where the scene has more than six and no more than eight) give the same bits: a block of particles at the largest size of a form, and with one particle more, far from all others."""
import numpy as np
import pytest

import sph_gb300
from scenes import lattice

pytestmark = pytest.mark.gpu

R = 0.01


@pytest.mark.parametrize("precision,per_sm", [("f32", 4 * 16), ("f32", 5 * 32), ("f64", 4 * 16), ("f64", 5 * 32), ("f64", 6 * 128), ("f64", 8 * 128)])
@pytest.mark.parametrize("lists", [64, 33, 24])
def test_lanes_give_the_same_bits(gpu_lib, precision, lists, per_sm):
    torch = pytest.importorskip("torch")
    n = torch.cuda.get_device_properties(0).multi_processor_count * per_sm
    side = int(np.ceil(n ** (1 / 3)))
    e = 2 * R * (side + 1) + 1e-9
    rng = np.random.default_rng(n)
    x = lattice(R, (2 * R,) * 3, (e,) * 3)[:n]
    x = np.vstack([x + rng.uniform(-0.2 * R, 0.2 * R, x.shape), [[e + 20 * R, e, e]]])
    v = np.vstack([rng.uniform(-0.2, 0.2, (n, 3)), np.zeros((1, 3))])
    b = sph_gb300.sample_box(4 * R, (0, 0, 0), (e + 2 * R,) * 3)
    out = []
    for m in (n, n + 1):
        s = sph_gb300.Scene(neighbor_list_max=lists, threads_per_particle=1, method=2, boundary=2, radius=R, precision=precision,
                            min_it=2, max_it=2, max_it_v=0, min_it_v=0, domain_min=(-4 * R,) * 3,
                            domain_max=(e + 30 * R,) * 3)
        s.set_fluid(x[:m], v[:m])
        s.add_boundary_points(b)
        s.init()
        out.append([s.get(f)[:n] for f in ("rho", "alpha")])
        s.step(1)
        q = s.pair_lists()
        out[-1] += [s.get(f)[:n] for f in ("rho", "alpha", "div", "v")] + [q["count"][:n], q["nbr"]]
    for a, w in zip(*out):
        assert np.array_equal(a, w)

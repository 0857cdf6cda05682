"""The pool's corrections load their records into registers, and from 1.2 M particles through a shared-memory ring: a
scene's results do not depend on which, nor on the solver shape."""
import numpy as np
import pytest

import sph_gb300
from scenes import lattice

pytestmark = pytest.mark.gpu

R = 0.01


def scene(side, seed):
    e = 2 * R * (side + 1) + 1e-9
    x = lattice(R, (2 * R,) * 3, (e,) * 3)
    rng = np.random.default_rng(seed)
    return (x + rng.uniform(-0.1 * R, 0.1 * R, x.shape), rng.uniform(-0.2, 0.2, x.shape),
            sph_gb300.sample_box(4 * R, (0, 0, 0), (e + 2 * R,) * 3))


def run(scenes, block, occupancy, lists):
    n, nb = sum(len(x) for x, _, _ in scenes), sum(len(b) for _, _, b in scenes)
    P = sph_gb300.Pool(max_particles=n, max_boundary=nb, max_keys=300_000 * len(scenes), max_scenes=len(scenes) + 1,
                       neighbor_list_max=lists)
    P.set_tuning(solver_block=block, solver_occupancy=occupancy)
    ids = [P.add_scene(x, v=v, boundary_points=b, steps=20, method=2, boundary=2, radius=R, precision="f32", eta=0.001, eta_v=0.001)
           for x, v, b in scenes]
    P.step(3)
    out = [P.get(ids[0], f) for f in ("x", "v", "rho", "k")]
    P.close()
    return n, out


@pytest.mark.parametrize("lists", [64, 30])
def test_record_forms_agree(gpu_lib, lists):
    first, other = scene(17, 1), scene(50, 2)
    n, want = run([first], 128, 1024, lists)
    assert n < 1_200_000
    for block, occupancy in ((128, 2048), (256, 1536)):
        for a, w in zip(run([first], block, occupancy, lists)[1], want):
            assert np.array_equal(a, w)
    for block in (128, 256):
        n, got = run([first] + [other] * 10, block, 1536, lists)
        assert n >= 1_200_000
        for a, w in zip(got, want):
            assert np.array_equal(a, w)

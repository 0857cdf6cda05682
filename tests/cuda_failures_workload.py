"""Scenarios of tests/test_cuda_failures_host.py: run in a process of its own with SPH_GB300_LIBRARY naming the library
linked against the fake CUDA runtime (tests/fake_cudart.cpp).  Prints one JSON line."""
import ctypes
import json
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import sph_gb300  # noqa: E402
from scenes import lattice  # noqa: E402

R = 0.02
FORCES = dict(visc_method=2, visc=0.01, bvisc=0.01, st_method=3, st=0.5, adh_method=4, adh=0.1)
SOLVERS = {
    "dfsph": dict(method=2), "dfsph_f64": dict(method=2, precision="f64"), "dfsph_forces": dict(method=2, **FORCES),
    "dfsph_walks": dict(method=2, neighbor_list_max=0, **FORCES), "wcsph": dict(method=0, visc_method=2, visc=0.01),
    "wcsph_forces": dict(method=0, **FORCES), "pcisph": dict(method=1, min_it=1, **FORCES),
}


def fake():
    return ctypes.CDLL(os.environ["SPH_GB300_LIBRARY"])


def scene(n_side=6, **p):
    s = sph_gb300.Scene(boundary=2, radius=R, **p)
    s.set_fluid(lattice(R, (2 * R,) * 3, (2 * R + 2 * R * n_side + 1e-9,) * 3))
    s.add_boundary_points(sph_gb300.sample_box(4 * R, (0, 0, 0), (0.6, 0.6, 0.6)))
    s.init()
    return s


def failed(call):
    try:
        call()
    except sph_gb300.SPHError:
        return True
    return False


def downloads(F):
    """A read whose staging buffer cannot be allocated fails; the next one works."""
    s = scene(**SOLVERS["dfsph"])
    P = sph_gb300.Pool(max_particles=1000, max_boundary=10_000, max_keys=100_000, max_scenes=2)
    P.set_autotune(0)
    P.set_graph(False)
    k = P.add_scene(lattice(R, (2 * R,) * 3, (0.3,) * 3), boundary_points=sph_gb300.sample_box(4 * R, (0, 0, 0), (0.6, 0.6, 0.6)),
                    steps=5, method=2, boundary=2, radius=R, precision="f32")
    P.step(1)
    out = {}
    for name, get in (("scene", s.get), ("pool", lambda f: P.get(k, f))):
        get("rho")
        F.fake_fail_malloc(1)  # x needs a larger buffer than rho
        first = failed(lambda: get("x"))
        out[name] = [first, failed(lambda: get("x")), failed(lambda: get("rho"))]
        out[name].append(failed(lambda: (s.step(1) if name == "scene" else P.step(1))))
    out["null_uses"] = F.fake_null_uses()
    return out


def launches(F):
    """Each launch of a step fails in turn: {solver: [launches, those whose failure the step did not report]}."""
    out = {}
    for name, p in SOLVERS.items():
        s = scene(**p)
        n0 = F.fake_launches()
        s.step(1)
        n = F.fake_launches() - n0
        lost = []
        for k in range(1, n + 1):
            F.fake_fail_launch(k)
            if not failed(lambda: s.step(1)):
                lost.append(k)
            F.fake_fail_launch(0)
        out[name] = [n, lost, failed(lambda: s.step(1))]
    return out


def allocations(F):
    """Each allocation of init fails in turn: {solver: [allocations, kernels of the candidate lists' build in a step,
    [those init did without, such kernels then launched in a step]]}."""
    out = {}
    for name, p in SOLVERS.items():
        def step():
            k = F.fake_launched(b"k_density_cand")
            scene(**p).step(1)
            return F.fake_launched(b"k_density_cand") - k

        m = F.fake_mallocs()
        lists = step()
        n = F.fake_mallocs() - m
        without = []
        for k in range(1, n + 1):
            F.fake_fail_malloc(k)
            try:
                without.append([k, step()])
            except sph_gb300.SPHError:
                pass
            F.fake_fail_malloc(0)
        out[name] = [n, lists, without]
    return out


def growth(F):
    """A particle leaves the grid box; each allocation of the growth that follows fails in turn: [growths, allocations],
    then per failure [the step reported it, growths, later steps failed]."""
    def grown(fail):
        s = scene(**SOLVERS["dfsph_forces"])
        F.fake_device_word(1)  # the escape flag, when the step polls it
        out, m = [], 0
        for k in range(40):
            m0 = F.fake_mallocs()
            if fail:
                F.fake_fail_malloc(fail)
            out.append(failed(lambda: s.step(1)))
            F.fake_fail_malloc(0)
            m = max(m, F.fake_mallocs() - m0)
            if F.fake_mallocs() > m0:  # it grew, or tried to
                break
        F.fake_device_word(0)
        later = any(failed(lambda: s.step(1)) for _ in range(3)) or failed(lambda: s.get("x"))
        return [any(out), s.stats()["grid_growths"], later, m]

    first = grown(0)
    return {"first": first, "each": [grown(k)[:3] for k in range(1, first[3] + 1)], "null_uses": F.fake_null_uses()}


if __name__ == "__main__":
    F = fake()
    print(json.dumps({"downloads": downloads, "launches": launches, "allocations": allocations, "growth": growth}[sys.argv[1]](F)))

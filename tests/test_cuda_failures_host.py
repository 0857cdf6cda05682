"""Failing allocations and launches, on the CPU: the library's own objects linked against a fake of the CUDA runtime
(tests/fake_cudart.cpp) that refuses a chosen one.

* A read whose staging buffer cannot be allocated reports it; later reads allocate again and nothing uses a null buffer.
* A step reports the failure of any of its launches.
* A scene whose candidate lists (or half-precision positions) find no memory runs without them.
* A grid box that finds no memory to grow stays as it is."""
import json
import os
import subprocess
import sys

import pytest

from sph_gb300 import buildlib

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.path.dirname(os.path.dirname(buildlib.nvcc()))


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    buildlib.build()
    objs = [os.path.join(buildlib.OBJDIR, os.path.splitext(u)[0] + ".o") for u in buildlib.UNITS]
    lib = str(tmp_path_factory.mktemp("fake") / "libsph_fake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(CUDA, "include"), "-o", lib,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-lpthread", "-ldl"], check=True, capture_output=True, text=True)

    def go(scenario):
        p = subprocess.run([sys.executable, os.path.join(HERE, "cuda_failures_workload.py"), scenario], capture_output=True,
                           text=True, timeout=300, env=dict(os.environ, SPH_GB300_LIBRARY=lib))
        assert p.returncode == 0, p.stderr[-2000:]
        return json.loads(p.stdout.strip().splitlines()[-1])

    return go


def test_failed_download_leaves_no_null_buffer(run):
    out = run("downloads")
    assert out["null_uses"] == 0
    for where in ("scene", "pool"):
        first, *later = out[where]
        assert first and not any(later), (where, out[where])


def test_step_reports_every_failed_launch(run):
    for solver, (n, lost, later) in run("launches").items():
        assert n >= 5 and lost == [] and not later, (solver, n, lost, later)


def test_scene_without_memory_for_candidate_lists(run):
    out = run("allocations")
    # half-precision positions of fluid and boundary; the lists and their two counts
    optional = {"dfsph": 2, "dfsph_f64": 2, "dfsph_forces": 5, "dfsph_walks": 0, "wcsph": 5, "wcsph_forces": 5, "pcisph": 5}
    for solver, (n, lists, without) in out.items():
        assert lists == (1 if optional[solver] == 5 else 0), solver
        assert without == [[k, 0] for k in range(n - optional[solver] + 1, n + 1)], (solver, n, without)


def test_grid_without_memory_to_grow(run):
    out = run("growth")
    failed, growths, later, n = out["first"]
    assert not failed and growths == 1 and not later and n >= 6
    assert out["null_uses"] == 0
    # the first is the staging buffer of the positions' download, whose failure the step reports
    assert out["each"][0] == [True, 0, False]
    for failed, growths, later in out["each"][1:]:
        assert not failed and not later and growths in (0, 1)

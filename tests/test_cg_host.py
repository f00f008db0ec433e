"""The host side of the device CG (``fne_cg_solve``, ``fne_cg_destroy``) on a stand-in for the CUDA runtime
(``cg_fake_runtime.cu``): which graphs it launches, what it records and waits for, failures included.  Runs on CPU."""

import math
import os
import shutil
import subprocess
from pathlib import Path

import pytest

from fenics_nonlinear_energies_b200 import _lib, build

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def solve(tmp_path_factory):
    nvcc = build._nvcc()
    if shutil.which(nvcc) is None:
        pytest.skip("needs nvcc")
    exe = tmp_path_factory.mktemp("cg") / "cg_host"
    out = subprocess.run([nvcc, "-O0", "-std=c++17", *build.ARCH, "-cudart", "none", "-o", os.fspath(exe),
                          os.fspath(HERE / "cg_fake_runtime.cu")], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-3000:]

    def run(*residuals, chunk=16, fail_graph=-1, fail_wait=-1, capturing=0):
        args = [chunk, fail_graph, fail_wait, capturing, *residuals]
        text = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, check=True, timeout=60).stdout
        head, calls, freed = text.splitlines()
        code, its, launches, told = map(int, head.split())
        return {"code": code, "its": its, "launches": launches, "told": told, "calls": calls.split(",")[:-1],
                "destroy": freed.split(",")}

    return run


@pytest.mark.parametrize("failure", [{}, {"fail_graph": 1}, {"fail_graph": 2}, {"fail_wait": 0}, {"fail_wait": 1}])
def test_end_of_work_is_recorded_on_every_way_out(solve, failure):
    """A solve that put work into the stream leaves the event that a later call on another stream, or the release
    of the handle, waits for -- also where a graph launch or a wait fails."""
    r = solve(1e-1, 1e-2, 1e-3, -1, **failure)
    assert r["code"] == (_lib.FNE_ECUDA if failure else _lib.FNE_OK)
    assert "graph" in r["calls"] and r["calls"][-1] == "record done"
    assert r["destroy"][0] == "wait done"


@pytest.mark.parametrize("residuals", [(-1,), (1e-1, -1), (1e-1, 1e-2, -1), (0.9, 0.8, 0.7, -1), (0.5, 1e-14, -1)])
def test_launches_count_the_graph_launched_ahead(solve, residuals):
    """The kernels a solve reports are those it launched, where the graph after the one with the stop was launched too."""
    r = solve(*residuals)
    assert r["its"] == 16 * len(residuals) and r["told"] == r["launches"]
    assert r["launches"] == 1 + 33 * r["calls"].count("graph")


def test_a_graph_ahead_is_launched_in_these_cases(solve):
    assert solve(0.9, 0.8, 0.7, -1)["calls"].count("graph") == 5
    assert solve(-1)["calls"].count("graph") == 1


@pytest.mark.parametrize("after_first", [math.nan, math.inf])
def test_no_graph_ahead_of_a_residual_without_a_rate(solve, after_first):
    """A residual that is not a number (or has overflowed) gives no rate to guess by: the next graph waits for the state."""
    calls = solve(after_first, -1)["calls"]
    assert calls == ["graph", "record ev0", "wait ev0", "graph", "record ev1", "wait ev1", "copy", "record done"]


def test_a_solve_under_capture_is_refused_before_it_leaves_anything(solve):
    """A solve is driven by the host, so it cannot be captured: nothing goes into the stream, the event least of all
    (a captured one would be refused by every later wait)."""
    r = solve(-1, capturing=1)
    assert r["code"] == _lib.FNE_ECUDA and r["calls"] == [] and r["launches"] == 0

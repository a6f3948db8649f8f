"""The host driver (the C ABI's host code) over a CUDA runtime on the CPU (tests/host/): what it hands to
kernels and copies, when it gives memory back, and what it does when a resource runs out."""
import os
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
UNITS = ["sst_api.cu", "sst_commit.cu", "sst_render.cu", "sst_adjoint_api.cu", "sst_query.cu"]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    from seesharp_gb300 import build
    cxx = shutil.which("g++")
    try:
        inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    except RuntimeError:
        pytest.skip("no CUDA toolkit")
    if cxx is None or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no g++ or no CUDA headers")
    out = tmp_path_factory.mktemp("host")
    sources = [os.path.join(build.CSRC, u) for u in UNITS] + [os.path.join(ROOT, "tests", "host", f) for f in ("fake_cuda.cpp", "driver_test.cpp")]

    def compile_unit(src):
        obj = str(out / (os.path.basename(src) + ".o"))
        subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-w", "-x", "c++", "-I", inc, "-I", os.path.join(ROOT, "include"), "-c", src, "-o", obj], check=True)
        return obj

    with ThreadPoolExecutor(len(sources)) as ex:
        objs = list(ex.map(compile_unit, sources))
    exe = str(out / "driver_test")
    subprocess.run([cxx, "-rdynamic", "-o", exe] + objs + ["-lpthread", "-ldl"], check=True)
    return exe


def run(driver, name, **env):
    p = subprocess.run([driver, name], capture_output=True, text=True, timeout=120, env={**os.environ, **env})
    assert p.returncode == 0, p.stdout + p.stderr


def test_query_job_table_is_uploaded_from_memory_that_stays(driver):
    run(driver, "query_job")


def test_results_may_overlay_the_rays(driver):
    run(driver, "overlay")


def test_renders_without_helper_threads(driver):
    run(driver, "threads")


def test_a_failed_render_has_waited_for_its_launches(driver):
    run(driver, "failed_render")


def test_unused_pool_memory_does_not_fail_allocations(driver):
    run(driver, "out_of_memory")


@pytest.mark.parametrize("megabytes", ["", "0", "100"])
def test_destroyed_scenes_leave_at_most_the_bound(driver, megabytes):
    run(driver, "scene_pool", **({"SST_SCENE_POOL_MB": megabytes} if megabytes else {}))


def test_large_batch_films_are_given_back(driver):
    run(driver, "batch_films")


def test_what_is_kept_does_not_depend_on_other_scenes(driver):
    run(driver, "several_scenes")

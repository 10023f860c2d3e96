"""Host-side failures (an allocation that throws, a CUDA call that fails) in
the library's C entries, by a program linked from the library's objects
(tests/cpp/failures.cpp): every one becomes a status code and gives back what
the call had taken."""
import importlib
import os
import subprocess

import pytest

from conftest import REPO

WRAPPED = ["cudaStreamCreateWithFlags", "cudaStreamDestroy", "cudaMallocFromPoolAsync", "cudaFreeAsync",
           "cudaMemPoolCreate", "cudaMemPoolSetAttribute", "cudaMemPoolTrimTo", "cudaMemPoolDestroy",
           "cudaMalloc", "cudaFree", "cudaMemcpy", "cudaMemGetInfo", "cudaGetDevice", "cudaDeviceSynchronize"]


@pytest.fixture(scope="module")
def program(pkg, tmp_path_factory):
    B = importlib.import_module("3dgrt_kdtree_gb300.build")
    units = [*B.CU_UNITS, *B.CPP_UNITS]
    objs = [os.path.join(B.OUT_DIR, u + ".o") for u in units]
    if not all(os.path.exists(o) for o in objs):
        B.build()
    exe = tmp_path_factory.mktemp("failures") / "failures"
    home = B._cuda_home()
    subprocess.run([os.path.join(home, "bin", "nvcc"), *B.ARCH, "-std=c++17", "-O1", "-I" + os.path.join(REPO, "include"),
                    "-I" + B.CSRC, os.path.join(REPO, "tests", "cpp", "failures.cpp"), *objs,
                    "-Xlinker", ",".join("--wrap=" + w for w in WRAPPED), "-lpthread", "-o", str(exe)], check=True)

    def run(case):
        r = subprocess.run([str(exe), case], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, f"{case}: exit {r.returncode}\n{r.stdout}{r.stderr}"

    return run


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["build_alloc", "build_alloc_threads"])
def test_device_build_allocations(program, cuda, case):
    program(case)


def test_shutdown_gives_back_every_pool(program):
    program("shutdown_pools")


def test_secondary_scene_allocations(program):
    program("secondary_alloc")


@pytest.mark.gpu
def test_scene_allocations(program, cuda):
    program("scene_alloc")


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["scene_room", "scene_share"])
def test_plain_leaf_order_takes_spare_memory_only(program, cuda, case):
    program(case)

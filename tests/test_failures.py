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


def link(source, exe, wrapped=()):
    """A program of tests/cpp, linked with the library's objects."""
    B = importlib.import_module("3dgrt_kdtree_gb300.build")
    objs = [os.path.join(B.OUT_DIR, u + ".o") for u in [*B.CU_UNITS, *B.CPP_UNITS]]
    if not all(os.path.exists(o) for o in objs):
        B.build()
    home = B._cuda_home()
    wrap = ["-Xlinker", ",".join("--wrap=" + w for w in wrapped)] if wrapped else []
    subprocess.run([os.path.join(home, "bin", "nvcc"), *B.ARCH, "-std=c++17", "-O1",
                    "-I" + os.path.join(REPO, "include"), "-I" + B.CSRC,
                    os.path.join(REPO, "tests", "cpp", source), *objs, *wrap, "-lpthread", "-o", str(exe)], check=True)
    return str(exe)


@pytest.fixture(scope="module")
def program(pkg, tmp_path_factory):
    exe = link("failures.cpp", tmp_path_factory.mktemp("failures") / "failures", WRAPPED)

    def run(case):
        r = subprocess.run([exe, case], capture_output=True, text=True, timeout=300)
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

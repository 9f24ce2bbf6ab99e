"""The block pool behind tl_alloc / tl_free (torchlette_b200/csrc/tl_pool.cu) without a GPU: linked against a fake of the CUDA calls
that it makes (tests/pool_stub/stub_cuda.cpp), which counts them and can make them fail."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "torchlette_b200", "csrc")
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pool") / "pool_stub_test")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-O1", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-x", "c++",
                    os.path.join(CSRC, "tl_pool.cu"), os.path.join(ROOT, "tests", "pool_stub", "stub_cuda.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("name", ["reuse", "failing_fence", "no_memory_for_the_fence", "bounds", "short_of_memory"])
def test_block_pool(harness, name):
    subprocess.run([harness, name], check=True)

"""The library's host side on the CPU: idb_api.cu compiled by g++ with a stand-in for
the CUDA runtime whose asynchronous work runs as late as the runtime's contract
allows and whose allocations can fail (tests/cpp/fake_cuda.hpp), under the address
sanitizer."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CPP = os.path.join(ROOT, "tests", "cpp")


def _cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("api_host") / "test_api_host")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-Wno-subobject-linkage", "-I" + _cuda_include(),
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "immunodbscan_gb300", "csrc"),
                    os.path.join(CPP, "test_api_host.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("name", ["tables_outlive_their_copies", "batch_run_with_more_genes_in_use",
                                  "buckets_when_the_join_does_not_fit", "side_records_decide",
                                  "candidates_by_pairs", "repeated_sweeps_keep_the_stamp", "long_eps_table"])
def test_api_host(exe, name):
    r = subprocess.run([exe, name], capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, ASAN_OPTIONS="detect_leaks=0"))
    assert r.returncode == 0, r.stdout + r.stderr

"""Rules of the kernels that need no device, compiled for the host from
csrc/device_common.cuh."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cpp") / "rules")
    subprocess.run([NVCC, "-gencode=arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "parallel-si_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "device_rules.cu"), "-o", out], check=True)
    return lambda name: subprocess.run([out, name], capture_output=True, text=True)


def test_barrier_words_past_four_billion_barriers(rules):
    r = rules("phases")
    assert r.returncode == 0, r.stdout


def test_the_evaluation_numbered_zero_is_a_full_one(rules):
    r = rules("numbers")
    assert r.returncode == 0, r.stdout


def test_walks_store_landmark_records_whole():
    """Walks read each other's records in the launch that writes them."""
    src = open(os.path.join(ROOT, "parallel-si_gb300", "csrc", "root_kernels.cu")).read()
    walks = src[src.index("k_root_walk(EvalArgs a)"):]
    assert "load_whole(&a.skip[" in walks and "store_whole(&a.skip[" in walks
    assert not re.search(r"a\.skip\[\w+\]\s*=[^=]", walks)

"""Which FP32 products are split for the tensor cores, and into what items: checked on
the host over all forms."""
import os
import subprocess

from conftest import PACKAGE, REPO

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_items_of_split_products(tmp_path):
    program = str(tmp_path / "gemm_split_plan_check")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(PACKAGE, "csrc"),
                    "-I", os.path.join(CUDA, "include"),
                    os.path.join(REPO, "tests", "gemm_split_plan_check.cpp"), "-o", program],
                   check=True)
    done = subprocess.run([program], stdout=subprocess.PIPE)
    assert done.returncode == 0, done.stdout.decode()[:2000]

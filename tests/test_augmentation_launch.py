"""Which kernels a batch's augmentation takes, what scratch they get and what becomes of
one that cannot be launched, on the host: the launch code compiled against stand-ins for the runtime's device calls."""
import os
import subprocess

from conftest import PACKAGE, REPO


def test_routes_scratch_and_failures(tmp_path):
    program = str(tmp_path / "augmentation_launch_check")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-cudart", "shared", "-I", os.path.join(PACKAGE, "csrc"),
                    os.path.join(REPO, "tests", "augmentation_launch_check.cpp"),
                    os.path.join(PACKAGE, "csrc", "augmentation.cu"), "-o", program],
                   check=True)
    done = subprocess.run([program], stdout=subprocess.PIPE)
    assert done.returncode == 0, done.stdout.decode()

"""Limits of dynamic shared memory follow the device a kernel is launched on (a
process may enable backends on several devices in turn), checked against a stand-in
for the CUDA runtime; and no launch site keeps such a limit once per process."""
import glob
import os
import re
import subprocess

from conftest import PACKAGE, REPO

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_limits_are_raised_on_every_device(tmp_path):
    program = str(tmp_path / "shared_limit_check")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(PACKAGE, "csrc"),
                    "-I", os.path.join(CUDA, "include"),
                    os.path.join(REPO, "tests", "shared_limit_check.cpp"), "-o", program],
                   check=True)
    done = subprocess.run([program], stdout=subprocess.PIPE)
    assert done.returncode == 0, done.stdout.decode()


def test_no_launch_site_keeps_a_limit_per_process():
    for path in glob.glob(os.path.join(PACKAGE, "csrc", "*.cu")):
        with open(path) as source:
            text = source.read()
        kept = re.findall(r"static[^;{]*cudaFuncSetAttribute|static bool configured", text)
        assert not kept, (path, kept)

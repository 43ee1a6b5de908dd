"""The epilogue warps of a tensor-core product write their staging blocks by their number,
whatever the launch set aside for them: too little (a tuning switch once gave eight warps
the room of four) is a write out of range, which no test may provoke.  So the host
arithmetic that sets it aside is what is checked, over every tile, epilogue and switch."""
import os
import re
import subprocess

from conftest import PACKAGE, REPO


def test_every_warp_has_its_staging(tmp_path):
    program = str(tmp_path / "gemm_tc_shared_check")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(PACKAGE, "csrc"),
                    os.path.join(REPO, "tests", "gemm_tc_shared_check.cpp"), "-o", program],
                   check=True)
    done = subprocess.run([program], stdout=subprocess.PIPE)
    assert done.returncode == 0, done.stdout.decode()[:2000]


def test_launches_take_that_arithmetic():
    with open(os.path.join(PACKAGE, "csrc", "gemm_tc.cu")) as source:
        text = source.read()
    assert re.findall(r"p\.staging_bytes = ([^;]*);", text) == ["shared.staging_bytes"]
    assert re.findall(r"p\.stages = ([^;]*);", text) == ["shared.stages"]
    assert re.findall(r"out->smem_bytes = ([^;]*);", text) == ["shared.bytes()"]
    assert "kTwoGroups = tc_two_groups(TILE_M, TILE_N, SECOND);" in text

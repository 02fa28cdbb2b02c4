"""The closed form of the FP64 push's segment cloud (csrc/segment_cloud.h), on the host."""
import os
import subprocess

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "cpp", "test_segment_cloud.cpp")


def test_closed_form(tmp_path):
    exe = str(tmp_path / "test_segment_cloud")
    subprocess.run(["g++", "-std=gnu++17", "-O2", "-ffp-contract=off", SRC, f"-I{ROOT}/scdat_b200/csrc", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

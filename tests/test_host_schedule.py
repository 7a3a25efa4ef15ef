"""The tile schedule's device code, run on the host by a small C++ program."""
import os
import subprocess

from conftest import ROOT
from graphic_lab_task_b200 import build as b


def test_host_schedule(tmp_path):
    exe = str(tmp_path / "host_schedule")
    subprocess.run(["g++"] + b.CXX_COMMON + [os.path.join(ROOT, "tests", "host_schedule.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[:2000]

"""Host builders of the derived layouts, checked by a small C++ program."""
import os
import subprocess

from conftest import ROOT
from graphic_lab_task_b200 import build as b


def test_host_layout(tmp_path):
    exe = str(tmp_path / "host_layout")
    subprocess.run(["g++"] + b.CXX_COMMON + [os.path.join(ROOT, "tests", "host_layout.cpp"),
                                             os.path.join(b.CSRC, "layout.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

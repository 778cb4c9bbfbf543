"""How ray batches are split over threads, up to the largest (a compiled check of the arithmetic; no device)."""
import os
import shutil
import subprocess

from conftest import ROOT


def test_every_ray_has_its_thread(tmp_path):
    exe = str(tmp_path / "trace_split")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Wextra", "-I", os.path.join(ROOT, "aurora_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "trace_split.cpp")], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout

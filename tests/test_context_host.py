"""Host code of the engine's context on a stand-in CUDA runtime (host memory, recorded launches; no GPU): C++
programs compiled here."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

DIR = os.path.join(ROOT, "tests", "context_check")
CSRC = os.path.join(ROOT, "johansen-null-eigenspectra_gb300", "csrc")


def _run(tmp_path, name, units=()):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if cxx is None or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path / name)
    srcs = [os.path.join(DIR, name + ".cpp"), *(os.path.join(CSRC, u) for u in units)]
    res = subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-Wno-attributes", "-isystem", cuda, "-x", "c++", *srcs, "-o", exe],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip().endswith("0 failures"), out.stdout[-2000:] + out.stderr[-2000:]


def test_tables_after_a_failed_allocation_or_upload(tmp_path):
    _run(tmp_path, "check_tables")


def test_launch_shapes_and_the_tuner(tmp_path):
    _run(tmp_path, "check_shapes", ["jne_api.cu", "jne_tune.cu"])


def test_order_of_a_ragged_launch(tmp_path):
    _run(tmp_path, "check_order")

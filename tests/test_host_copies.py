"""The staged host copies over a fake runtime (tests/fake/stage.cu), on the CPU."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "secure-vector-search_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def stage(tmp_path_factory):
    if not (os.path.exists(NVCC) or shutil.which(NVCC)):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("stage") / "stage")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xcompiler", "-fopenmp",
                    f"-I{CSRC}", f"-I{os.path.join(ROOT, 'include')}", os.path.join(ROOT, "tests", "fake", "stage.cu"),
                    "-o", exe], check=True)
    return exe


def test_two_threads_share_the_slots(stage):
    assert subprocess.run([stage, "copies"], timeout=120).returncode == 0


def test_failed_pinning_is_not_tried_on_every_copy(stage):
    """200 MB of copies, 64 MB of which repay the slots: three tries."""
    out = subprocess.run([stage, "pinfail"], timeout=120, capture_output=True, text=True)
    assert out.returncode == 0 and int(out.stdout) == 3

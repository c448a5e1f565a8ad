"""The one-launch builder when its grid's wait runs out: an error status, a usable context and a
good next build.  The program sets the limit to nothing, so that no CTA waits at all."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_is_reported(tmp_path):
    exe = str(tmp_path / "small_wait")
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "fakes", "small_wait.cu"), os.path.join(PKG, "csrc", "small.cu"),
                    os.path.join(PKG, "csrc", "devmem.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "small wait ok" in out.stdout, out.stdout + out.stderr

"""CPU checks of the library's memory bookkeeping (csrc/devmem.cu, the handle's release) and of
what it does with a refused launch, on a host-side CUDA runtime of two devices (tests/fakes): no
GPU is touched."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import PKG, ROOT

CHECKS = ["handle_of_another_device", "buffer_of_another_device", "arrays_of_another_device",
          "slots_of_many_threads", "slots_across_a_reset", "contexts_in_turn", "opt_ins", "refused_launch", "trim"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("devmem") / "devmem_check"
    fakes = os.path.join(ROOT, "tests", "fakes")
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "none",
                    "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"), "-I", fakes,
                    os.path.join(fakes, "devmem_check.cu"), os.path.join(fakes, "cudart.cpp"), os.path.join(PKG, "csrc", "devmem.cu"),
                    os.path.join(PKG, "csrc", "small.cu"),
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("check", CHECKS)
def test_devmem(program, check):
    out = subprocess.run([program, check], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr

"""The correctly rounded operations of the fast physics (csrc/mhd_fast.cuh) on
the GPU, from its own reciprocal and root approximations: the operands of
tests/test_fast_physics_cpu.py, where the host's truncated quotients stand in
for them."""
from __future__ import annotations

import ctypes as C
import subprocess

import pytest

import test_fast_physics_cpu as cpu
from athena_cuda_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fast(tmp_path_factory):
    so = tmp_path_factory.mktemp("fast") / "libfast_device.so"
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-shared", f"-I{build.CSRC}", "-o", str(so),
                    str(cpu.HERE / "hostcheck" / "fast_device.cu")], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("check", [cpu.test_reciprocals_correctly_rounded, cpu.test_quotients_correctly_rounded,
                                   cpu.test_roots_correctly_rounded, cpu.test_operations_at_the_ends_of_their_ranges])
def test_operations_on_the_gpu(fast, check):
    check(fast)

"""A product wait of the complex64 block kernels that gives up: the group whose
wait it was leaves as one, the other group of its CTA finishes its tiles, and
the kernel returns (tests/cxx/block_wait.cu)."""
import os
import subprocess

import pytest

from kate_b200 import build as B

pytestmark = pytest.mark.gpu
SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cxx", "block_wait.cu")


def test_a_wait_that_gives_up_ends_its_group_only(tmp_path):
    exe = str(tmp_path / "block_wait")
    subprocess.run([B.NVCC, *B.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-DKATE_BLOCK_WAIT_LIMIT=1024",
                    "-I" + B.CSRC, "-I" + os.path.join(B.ROOT, "include"), SRC, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    want = [f"lost {lost} group {g}: gave up {lost >> g & 1} tiles {0 if lost >> g & 1 else 5}"
            for lost in range(4) for g in range(2)] + ["disagreements 0"]
    assert r.stdout.splitlines() == want, r.stdout + r.stderr
    assert r.returncode == 0

"""The bounded waits of the tensor-core kernels (csrc/tests/wait_check.cu, csrc/tcgen05.cuh): given up at their limit by the clock."""
import subprocess

import pytest
import torch

from tensorsharp_b200.ops import native


def _exe():
    return str({p.name: p for p in native.build_tests()}["wait_check"])


def test_wait_check_builds_and_skips_without_a_gpu():
    exe = _exe()
    if torch.cuda.is_available():
        pytest.skip("GPU present: covered by the gpu test")
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 77 and "SKIP" in p.stdout


@pytest.mark.gpu
def test_waits_end_at_their_limit():
    p = subprocess.run([_exe()], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip().endswith("OK"), p.stdout + p.stderr

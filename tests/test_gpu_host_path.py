"""The native host path of the Python entry points at its edges: calls that it must leave to the Python path, or must not change."""
import subprocess
import sys

import pytest
import torch

import kiln_b200

pytestmark = pytest.mark.gpu


def _child(code):
    """Runs code in a process of its own (what it tests would end the process) and returns its output."""
    done = subprocess.run([sys.executable, "-c", "import torch, kiln_b200\ndev = torch.device('cuda')\n" + code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, f"exit code {done.returncode}\n{done.stderr[-2000:]}"
    return done.stdout


def test_a_problem_without_rows_of_weights_is_refused(cuda_device):
    out = _child("""
try:
    kiln_b200.marlin_w4a16_gemm(torch.empty((4, 0), dtype=torch.bfloat16, device=dev), torch.empty((0, 512), dtype=torch.int32, device=dev),
                                torch.empty((0, 256), dtype=torch.float16, device=dev), 128)
except kiln_b200.KilnMarlinError as e:
    print(e)
""")
    assert "k=0 must be divisible by groupsize=128" in out

"""The first AUTO call of a size: where the tensor cores beat even the FMA
pipe's peak, no FMA kernel is timed."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys
sys.path.insert(0, sys.argv[1])
import torch, gbblas
A, B, C = (torch.zeros(2048, 2048, device="cuda") for _ in range(3))
def launches():
    n = gbblas.kernel_launches()
    gbblas.gemm(A, B, C, accuracy=gbblas.ACCURACY_AUTO)
    torch.cuda.synchronize()
    return gbblas.kernel_launches() - n
first, then = launches(), launches()
assert then > 1, "AUTO took the FMA pipe"
assert first == 5 * then, (first, then)  # a warm-up, three timed, the call itself
"""


def test_first_auto_call_times_the_tensor_cores_alone(cuda, tmp_path):
    env = {k: v for k, v in os.environ.items() if not k.startswith("GBBLAS_")}
    env["GBBLAS_TUNE_CACHE"] = str(tmp_path / "tune.json")
    r = subprocess.run([sys.executable, "-c", CODE, os.path.join(ROOT, "openmp-blas_gb300")], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "gemm_fma_tile|" not in (tmp_path / "tune.json").read_text()

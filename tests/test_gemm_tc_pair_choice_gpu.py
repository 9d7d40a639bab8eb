"""A bucket whose tuned choice is CTA pairs: a product whose C does not admit
pairs (contiguous rows off the 16-byte grid) takes single CTAs and the K parts
that the rule gives it, as it does where nothing is tuned."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import os, sys
sys.path.insert(0, sys.argv[1])
import torch, gbblas
M, N, K = 512, 256, 8192
A, B = torch.rand(M, K, device="cuda") - 0.5, torch.rand(K, N, device="cuda") - 0.5

def launches(ldc, fixed=None):
    C = torch.zeros(M, ldc, device="cuda")[:, :N]
    if fixed:
        os.environ["GBBLAS_TC_SPLITK"] = fixed
    gbblas.gemm(A, B, C, accuracy=gbblas.ACCURACY_BF16X6)  # set-up and scratch
    n = gbblas.kernel_launches()
    gbblas.gemm(A, B, C, accuracy=gbblas.ACCURACY_BF16X6)
    os.environ.pop("GBBLAS_TC_SPLITK", None)
    return gbblas.kernel_launches() - n, C

plain, want = launches(N + 1, "1")
pair, _ = launches(N)
cut, got = launches(N + 1)
assert pair == plain, "the cache was not read"
assert cut == plain + 1, "the parts' reduction is missing"
exact = 2 * (A.double() @ B.double())
mag = 2 * (A.abs().double() @ B.abs().double())
assert bool(((got.double() - exact).abs() <= 4 * K * 2.0 ** -23 * mag).all())
"""


def test_no_pairs_keeps_the_split(cuda, tmp_path):
    p = cuda.cuda.get_device_properties(0)
    tag = f"{p.name.replace(' ', '_')}_sm{p.multi_processor_count}"
    cache = tmp_path / "tune.json"
    cache.write_text(json.dumps({"version": 1, f"gemm_tc|{tag}|mode3|m9|n8|k13|pair": 1}))
    env = {k: v for k, v in os.environ.items() if k not in ("GBBLAS_TC_PAIR", "GBBLAS_TC_SPLITK")}
    env["GBBLAS_TUNE_CACHE"] = str(cache)
    r = subprocess.run([sys.executable, "-c", CODE, os.path.join(ROOT, "openmp-blas_gb300")], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

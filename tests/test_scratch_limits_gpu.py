"""Calls whose scratch does not fit: what only makes a call faster is left out
and the call still runs.  Each runs in a process of its own whose memory pool
(what the library's scratch comes from) holds 32 MB."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import torch, gbblas

def limit_pool():
    class Location(ctypes.Structure):
        _fields_ = [("type", ctypes.c_int), ("id", ctypes.c_int)]
    class Props(ctypes.Structure):
        _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("location", Location),
                    ("security", ctypes.c_void_p), ("maxSize", ctypes.c_size_t), ("usage", ctypes.c_ushort),
                    ("reserved", ctypes.c_ubyte * 54)]
    cu, pool = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p()
    props = Props(allocType=1, location=Location(1, 0), maxSize=32 << 20)
    assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    assert cu.cuDeviceSetMemPool(0, pool) == 0

def run(stream, A, B, C0, accuracy):
    C = C0.clone()
    torch.cuda.synchronize()
    gbblas.gemm(A, B, C, accuracy=accuracy, stream=stream)
    gbblas.call("gbblas_check_stream", stream.cuda_stream)
    return C

def operands(M, N, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M)
    return [torch.rand(s, generator=g, device="cuda", dtype=dtype) * 2 - 1 for s in ((M, K), (K, N), (M, N))]
"""


def child(code):
    r = subprocess.run([sys.executable, "-c", PRELUDE + code, os.path.join(ROOT, "openmp-blas_gb300")], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("accuracy", [3, 6])  # AUTO, DIGITS7
def test_digit_gemm_without_room_for_the_cut(cuda, accuracy):
    """23 (20) MB of digit planes, 12 (10) of slots for the last tiles' parts,
    allocated with a quarter on top."""
    child(f"""
ops = operands(512, 608, 1280, torch.float64)
want = run(torch.cuda.Stream(), *ops, {accuracy})
limit_pool()
s = torch.cuda.Stream()
n = gbblas.kernel_launches()
got = run(s, *ops, {accuracy})
assert torch.equal(got, want)
assert gbblas.kernel_launches() - n >= 4, "not the digits"
""")


@pytest.mark.parametrize("accuracy", ["ACCURACY_AUTO", "ACCURACY_FP16X3"])
def test_tensor_core_gemm_without_room_for_the_parts(cuda, accuracy):
    """20 MB of FP16 pieces, 8 of partial sums for K in two parts."""
    child(f"""
import os
acc = gbblas.{accuracy}
os.environ["GBBLAS_GEMM_AUTO"] = "1"
ops = operands(1024, 1024, 2400, torch.float32)
os.environ["GBBLAS_TC_SPLITK"] = "1"
want = run(torch.cuda.Stream(), *ops, acc)
del os.environ["GBBLAS_TC_SPLITK"]
cut = run(torch.cuda.Stream(), *ops, acc)
assert not torch.equal(cut, want), "K is not cut here"
limit_pool()
assert torch.equal(run(torch.cuda.Stream(), *ops, acc), want)
""")

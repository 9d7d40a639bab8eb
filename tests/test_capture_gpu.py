"""Single calls recorded into a caller's CUDA graph: a call whose scratch its
stream already holds records its own kernels only - nothing is timed, also
where it is the first of its shape - and every replay does what the call does."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_first_auto_call_of_a_shape_times_nothing(cuda, tmp_path):
    """With nothing tuned yet (an empty cache, a process of its own)."""
    code = """
import sys
sys.path.insert(0, sys.argv[1])
import torch, gbblas
A, B, C = (torch.rand(s, device="cuda") - 0.5 for s in ((700, 800), (800, 900), (700, 900)))
out = C.clone()
s = torch.cuda.Stream()
torch.cuda.synchronize()
gbblas.gemm(A, B, out, accuracy=gbblas.ACCURACY_FP16X3, stream=s)  # the library's set-up and the stream's scratch
out.copy_(C)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
n = gbblas.kernel_launches()
with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
    gbblas.gemm(A, B, out, accuracy=gbblas.ACCURACY_AUTO)
n = gbblas.kernel_launches() - n
assert 1 <= n <= 8, f"{n} kernels launched by one call"
out.copy_(C)
torch.cuda.synchronize()
g.replay()
torch.cuda.synchronize()
err = (out.double() - (C.double() + A.double() @ B.double())).abs()
mag = C.abs().double() + A.abs().double() @ B.abs().double()
assert bool((err <= 2 * 800 * 2.0 ** -23 * mag).all())
"""
    env = dict(os.environ, GBBLAS_TUNE_CACHE=str(tmp_path / "tune.json"))
    env.pop("GBBLAS_AUTOTUNE", None)
    r = subprocess.run([sys.executable, "-c", code, os.path.join(ROOT, "openmp-blas_gb300")], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


# chains: tables by tc_init_kernel, K cut along with the parts' reduction and
# the guard's fix-up; digits with cut tiles; GEMVs with a chained finish
CALLS = ["auto", "auto_cut", "bf16x3", "fp8", "double", "mtv_rows", "mtv_columns", "mtv_columns_double"]


@pytest.mark.parametrize("name", CALLS)
def test_replays_do_what_the_call_does(cuda, name, monkeypatch):
    import gbblas
    torch = cuda
    dt = torch.float64 if "double" in name else torch.float32
    g = torch.Generator(device="cuda").manual_seed(len(name))
    rand = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=dt) - 0.5  # noqa: E731
    if name.startswith("mtv"):
        # rows of 40001 in several ranges, columns in more than eight
        layout, M, N = (gbblas.LAST_ORDER, 37, 400001) if name == "mtv_rows" else (gbblas.FIRST_ORDER, 1001, 6001)
        ins = [rand(M, N) if layout else rand(N, M), rand(N)]
        out0, call = rand(M), lambda o: gbblas.mtv(layout, M, N, ins[0], ins[1], o)
    else:
        M, N, K = {"auto_cut": (300, 200, 4000), "double": (300, 100, 1100)}.get(name, (513, 400, 700))
        ins = [rand(M, K), rand(K, N)]
        accuracy = {"bf16x3": gbblas.ACCURACY_BF16X3, "fp8": gbblas.ACCURACY_FP8,
                    "double": gbblas.ACCURACY_FP32}.get(name, gbblas.ACCURACY_AUTO)
        monkeypatch.setenv("GBBLAS_GEMM_AUTO", "1")
        out0, call = rand(M, N), lambda o: gbblas.gemm(ins[0], ins[1], o, accuracy=accuracy)
    others = [torch.roll(t, 1, 0).contiguous() for t in ins]
    s, out = torch.cuda.Stream(), out0.clone()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        call(out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call(out)
    for values in ([t.clone() for t in ins], others, others):
        for t, v in zip(ins, values):
            t.copy_(v)
        out.copy_(out0)
        want = out0.clone()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            call(want)
        torch.cuda.synchronize()
        assert torch.equal(out, want)

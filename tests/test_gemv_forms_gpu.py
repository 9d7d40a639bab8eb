"""GEMV at the edges of its launch forms: the short rows (a warp each), one and
four rows a group, the large float matrices of three CTAs an SM, columns by
single rows, by vectors and by shifted vectors."""
import pytest

from _tol import C_GEMM, eps

pytestmark = pytest.mark.gpu

SHORT = [(m, n) for m in (1, 7, 9, 1023, 1024, 1025) for n in (1, 3, 127, 255, 256, 257, 511, 512, 513)]
ROWS = [(1024, 2050), (1027, 1029), (2999, 515), (3000, 516), (3005, 1031), (613, 4096), (700, 3000), (153, 9000),
        (4101, 20000), (4100, 20003)]
COLS = [(2047, 33), (2049, 513), (5003, 999), (5004, 1001), (7001, 4001), (7003, 3200)]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("layout,M,N", [(1, *s) for s in SHORT + ROWS] + [(0, *s) for s in COLS])
@pytest.mark.parametrize("off", [0, 1])
def test_forms(cuda, dtype, layout, M, N, off):
    """Against the same product in 64 bits (128 in sum for double: by columns),
    off the 16-byte grid by `off` elements, guarded by NaN; twice, same bits."""
    import gbblas
    torch = cuda
    dt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    flat = torch.full((M * N + off + 4,), float("nan"), device="cuda", dtype=dt)
    flat[off:off + M * N] = torch.rand(M * N, generator=g, device="cuda", dtype=dt) * 2 - 1
    x = torch.full((N + off + 4,), float("nan"), device="cuda", dtype=dt)
    x[off:off + N] = torch.rand(N, generator=g, device="cuda", dtype=dt) * 2 - 1
    A = flat[off:off + M * N].view(M, N) if layout else flat[off:off + M * N].view(N, M).t()
    out = []
    for _ in range(2):
        y = torch.full((M + 3,), float("nan"), device="cuda", dtype=dt)
        gbblas.call(f"gbblas_{'s' if dt is torch.float32 else 'd'}gemv", layout, 0, M, N, flat[off:].data_ptr(),
                    x[off:].data_ptr(), 0, y.data_ptr(), None)
        assert bool(torch.isnan(y[M:]).all())
        out.append(y[:M])
    assert torch.equal(out[0], out[1])
    e = eps("float32" if dt is torch.float32 else "float64")
    for r in range(0, M, 1024):  # the scale, and the reference, in pieces
        a = A[r:r + 1024].double()
        exact, scale = a @ x[off:off + N].double(), a.abs() @ x[off:off + N].double().abs()
        # (in double the reference's own error counts too: as many roundings again)
        k = N if dt is torch.float32 else 2 * N
        assert bool(((out[0][r:r + 1024].double() - exact).abs() <= C_GEMM * k * e * scale).all())

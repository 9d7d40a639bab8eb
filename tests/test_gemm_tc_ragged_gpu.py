"""Tensor-core GEMMs whose operands and results sit at awkward places: odd
leading dimensions, bases off the 16-byte grid, extents that are multiples of
nothing.  Each case computes the same product from the same values as an
aligned call, so the results must agree bit for bit, and the memory around C
must stay as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BF16X3, FP8, BF16X6, FP16X3 = 1, 2, 4, 8


def place(torch, X, pitch, off, col_major=False, step=1):
    """X (numpy, 2-D) in a device buffer: row (column) pitch `pitch`, first
    element at `off`, neighbours `step` apart; returns (buffer, address, row
    stride, column stride, the elements' places, their shape)."""
    v = X.T if col_major else X
    buf = np.full(off + v.shape[0] * pitch * step + 7, np.float32(-77.0), np.float32)
    at = (off + np.arange(v.shape[0])[:, None] * pitch * step + np.arange(v.shape[1])[None, :] * step).ravel()
    buf[at] = v.ravel()
    t = torch.from_numpy(buf).cuda()
    rs, cs = (step, pitch * step) if col_major else (pitch * step, step)
    return t, t.data_ptr() + 4 * off, rs, cs, at, v.shape


def gemm(torch, A, B, C0, acc, pa, pb, pc, la=False, lb=False, lc=False):
    import gbblas
    M, K = A.shape
    N = B.shape[1]
    a = place(torch, A, (M if la else K) + pa[0], pa[1], la, *pa[2:])
    b = place(torch, B, (K if lb else N) + pb[0], pb[1], lb, *pb[2:])
    c = place(torch, C0, (M if lc else N) + pc[0], pc[1], lc)
    gbblas.call("gbblas_sgemm", M, N, K, a[1], a[2], a[3], b[1], b[2], b[3], c[1], c[2], c[3], acc, None)
    gbblas.call("gbblas_check_stream", None)
    out = c[0].cpu().numpy()
    rest = np.ones(out.size, bool)
    rest[c[4]] = False
    assert np.all(out[rest] == np.float32(-77.0)), "memory beside C changed"
    got = out[c[4]].reshape(c[5])
    return got.T if lc else got


def values(rng, shape):
    return rng.uniform(-1, 1, shape).astype(np.float32)


# C rows: aligned (the TMA update), pitches and bases that are not (the
# warp-by-row update); extents at the tile's edges
@pytest.mark.parametrize("acc", [BF16X3, FP8, BF16X6, FP16X3])
@pytest.mark.parametrize("M,N,K", [(1, 4, 8), (127, 132, 64), (128, 128, 128), (129, 260, 520), (33, 700, 260)])
@pytest.mark.parametrize("pad,off", [(1, 0), (2, 0), (3, 3), (0, 1)])
def test_unaligned_c_same_bits_as_aligned(cuda, acc, M, N, K, pad, off):
    rng = np.random.default_rng(M * 7 + N + K)
    A, B, C0 = values(rng, (M, K)), values(rng, (K, N)), values(rng, (M, N))
    want = gemm(cuda, A, B, C0, acc, (0, 0), (0, 0), (0, 0))
    got = gemm(cuda, A, B, C0, acc, (0, 0), (0, 0), (pad, off))
    np.testing.assert_array_equal(got, want)


# Operands: every preparation route (K contiguous at 16-, 8- and 4-byte
# aligned rows, one pass per row or per warp; rows contiguous, aligned or not)
# against the strided tile route (neighbours two apart) on the same values
@pytest.mark.parametrize("acc", [BF16X3, BF16X6, FP16X3, FP8])
@pytest.mark.parametrize("M,N,K", [(130, 135, 1), (129, 260, 67), (140, 1030, 1023), (65, 129, 1025), (40, 30, 8191),
                                   (16, 20, 8200)])
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (2, 2), (3, 1)])
@pytest.mark.parametrize("cols", [False, True])
def test_operand_routes_same_bits(cuda, acc, M, N, K, pad, off, cols):
    rng = np.random.default_rng(M + N * 3 + K)
    A = (values(rng, (M, K)) * np.float32(2.0) ** rng.integers(-6, 7, (M, K))).astype(np.float32)
    B = (values(rng, (K, N)) * np.float32(2.0) ** rng.integers(-6, 7, (K, N))).astype(np.float32)
    A[M // 2] = 0.0
    C0 = values(rng, (M, N))
    want = gemm(cuda, A, B, C0, acc, (0, 0, 2), (0, 0, 2), (0, 0), False, False)
    got = gemm(cuda, A, B, C0, acc, (pad, off), (pad, off), (0, 0), cols, not cols)
    np.testing.assert_array_equal(got, want)


# K cut into parts under AUTO's guard: outputs in out-of-span rows and columns
# are left out of the partials and computed once by the fix-up; everything
# stays inside the guard's bound (2^-19 + 2 K eps32) (|A||B|) plus the addition
# into C, and repeats bit for bit
@pytest.mark.parametrize("parts", [1, 2, 3, 16])
@pytest.mark.parametrize("M,N,K", [(40, 30, 1025), (129, 257, 4100), (300, 64, 2048)])
@pytest.mark.parametrize("lc", [False, True])
def test_split_k_under_the_guard(cuda, monkeypatch, parts, M, N, K, lc):
    monkeypatch.setenv("GBBLAS_GEMM_AUTO", "1")
    monkeypatch.setenv("GBBLAS_TC_SPLITK", str(parts))
    rng = np.random.default_rng(parts + M)
    A, B, C0 = values(rng, (M, K)), values(rng, (K, N)), values(rng, (M, N))
    A[M // 3] *= np.float32(2.0 ** -30)  # a row and a column whose magnitudes span too far
    A[M // 3, 0] = 1.0
    B[:, N // 2] *= np.float32(2.0 ** -30)
    B[0, N // 2] = 1.0
    got = gemm(cuda, A, B, C0, 3, (1, 0), (0, 0), (1, 0), False, False, lc)
    exact = A.astype(np.float64) @ B.astype(np.float64) + C0
    mag = np.abs(A).astype(np.float64) @ np.abs(B)
    assert np.all(np.abs(got - exact) <= (2.0 ** -19 + 2 * K * 2.0 ** -23) * mag + 2.0 ** -23 * (np.abs(C0) + mag))
    np.testing.assert_array_equal(gemm(cuda, A, B, C0, 3, (1, 0), (0, 0), (1, 0), False, False, lc), got)

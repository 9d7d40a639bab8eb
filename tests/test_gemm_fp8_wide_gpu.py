"""FP8 GEMMs large enough for the 128 x 256 tiles: the same bits as calls on
column slabs narrow enough for 128 x 128 tiles (both add the products in the
same order), exact on small integers, and nothing written beside C.  Extents
at the tiles' edges: a last tile with 6 columns in its second half, with none
there, K of part of a scale atom, of whole ones and of an odd count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP8 = 2
SLAB = 1000


def gemm(torch, A, B, C0, pad=0, col_c=False):
    import gbblas
    M, K = A.shape
    N = B.shape[1]
    V = C0.T if col_c else C0
    buf = torch.full((V.shape[0], V.shape[1] + pad), -77.0, device="cuda")
    buf[:, :V.shape[1]] = torch.from_numpy(np.ascontiguousarray(V))
    a, b = torch.from_numpy(A).cuda(), torch.from_numpy(np.ascontiguousarray(B)).cuda()
    ld = V.shape[1] + pad
    rs, cs = (1, ld) if col_c else (ld, 1)
    gbblas.call("gbblas_sgemm", M, N, K, a.data_ptr(), K, 1, b.data_ptr(), N, 1, buf.data_ptr(), rs, cs, FP8, None)
    gbblas.call("gbblas_check_stream", None)
    out = buf.cpu().numpy()
    assert np.all(out[:, V.shape[1]:] == np.float32(-77.0)), "memory beside C changed"
    got = out[:, :V.shape[1]]
    return got.T if col_c else got


@pytest.mark.parametrize("M,N", [(1500, 2900), (1410, 2950), (1536, 3072)])
@pytest.mark.parametrize("K", [1, 200, 512, 640, 2304])
@pytest.mark.parametrize("pad,col_c", [(0, False), (4, False), (1, False), (0, True)])
def test_wide_tiles_same_bits_as_narrow(cuda, M, N, K, pad, col_c):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A = rng.uniform(-1, 1, (M, K)).astype(np.float32) * np.exp2(rng.integers(-6, 7, (M, 1))).astype(np.float32)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float32) * np.exp2(rng.integers(-6, 7, (1, N))).astype(np.float32)
    A[:, 128:300] *= 2.0 ** 5  # scales that differ along K
    C0 = rng.uniform(-1, 1, (M, N)).astype(np.float32)
    want = np.concatenate([gemm(cuda, A, B[:, n:n + SLAB], C0[:, n:n + SLAB]) for n in range(0, N, SLAB)], axis=1)
    np.testing.assert_array_equal(gemm(cuda, A, B, C0, pad, col_c), want)


def test_wide_tiles_integers_exact(cuda):
    M, N, K = 1500, 2950, 700
    rng = np.random.default_rng(1)
    A = rng.integers(-8, 9, (M, K)).astype(np.float32)
    B = rng.integers(-8, 9, (K, N)).astype(np.float32)
    C0 = rng.integers(-50, 51, (M, N)).astype(np.float32)
    np.testing.assert_array_equal(gemm(cuda, A, B, C0), A.astype(np.float64) @ B + C0)


def test_wide_tiles_grouped(cuda):
    import gbblas
    rng = np.random.default_rng(2)
    descs, cs, want = [], [], []
    for M, N, K in [(700, 2900, 640), (40, 100, 300), (900, 3000, 300)]:
        A = rng.uniform(-1, 1, (M, K)).astype(np.float32)
        B = rng.uniform(-1, 1, (K, N)).astype(np.float32)
        want.append(gemm(cuda, A, B, np.zeros((M, N), np.float32)))
        a, b = cuda.from_numpy(A).cuda(), cuda.from_numpy(B).cuda()
        c = cuda.zeros((M, N), dtype=cuda.float32, device="cuda")
        cs.append((a, b, c))
        descs.append(gbblas.gemm_desc(a, b, c))
    gbblas.gemm_grouped(descs, accuracy=FP8)
    cuda.cuda.synchronize()
    for (_, _, c), w in zip(cs, want):
        np.testing.assert_array_equal(c.cpu().numpy(), w)

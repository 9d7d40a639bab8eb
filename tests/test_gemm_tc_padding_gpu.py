"""Split-BF16 operand preparation leaves the padding rows of an operand (up to
the next multiple of 128) as the scratch held them.  A call that fills the
scratch with NaN pieces before must not change a later call's result, whose
padding rows then hold NaN: extents around the tiles' edges, every layout of
the operands (row-by-row preparation, tiles with wide and with scalar loads)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BF16X3, BF16X6 = 1, 4


def gemm(torch, A, B, C0, acc, la, lb):
    import gbblas
    a = torch.from_numpy(np.ascontiguousarray(A if la else A.T)).cuda()
    b = torch.from_numpy(np.ascontiguousarray(B if lb else B.T)).cuda()
    c = torch.from_numpy(C0.copy()).cuda()
    gbblas.gemm(a if la else a.t(), b if lb else b.t(), c, accuracy=acc)
    torch.cuda.synchronize()
    return c.cpu().numpy()


@pytest.mark.parametrize("acc", [BF16X3, BF16X6])
@pytest.mark.parametrize("la,lb", [(1, 1), (0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (65, 129, 100), (100, 200, 520), (127, 132, 96), (300, 40, 61)])
def test_stale_nan_in_padding_rows(cuda, acc, la, lb, M, N, K):
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A = rng.integers(-8, 9, (M, K)).astype(np.float32)
    B = rng.integers(-8, 9, (K, N)).astype(np.float32)
    C0 = rng.integers(-50, 51, (M, N)).astype(np.float32)
    bad = np.full((1024, 1024), np.nan, np.float32)
    gemm(cuda, bad, bad, np.zeros((1024, 1024), np.float32), acc, la, lb)
    np.testing.assert_array_equal(gemm(cuda, A, B, C0, acc, la, lb), A.astype(np.float64) @ B + C0)

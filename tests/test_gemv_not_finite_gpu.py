"""Inf and NaN in GEMV: what a kernel reads beside a row or column to reach a
16-byte boundary, or puts in the place of elements that do not exist, never
meets them - only the outputs that hold such a term are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# both kernels; odd leading dimensions, off the 16-byte grid; first, last and
# inner row blocks, one and several splits
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("cols_form", [False, True])
@pytest.mark.parametrize("M,K", [(5, 3), (125, 65), (131, 1023), (700, 2047)])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_only_outputs_with_such_a_term(cuda, dt, cols_form, M, K, off):
    import gbblas
    torch = cuda
    rng = np.random.default_rng(M + K + off)
    size = np.dtype(dt).itemsize
    fn = f"gbblas_{'s' if dt == np.float32 else 'd'}gemv"

    def run(A, x):
        stored = (A.T if cols_form else A).ravel()
        buf = torch.from_numpy(np.concatenate([np.full(off, np.nan, dt), stored, np.full(5, np.nan, dt)])).cuda()
        tx, ty = torch.from_numpy(x).cuda(), torch.zeros(M, dtype=torch.from_numpy(x).dtype, device="cuda")
        gbblas.call(fn, 0 if cols_form else 1, 0, M, K, buf.data_ptr() + off * size, tx.data_ptr(), 1, ty.data_ptr(), None)
        return ty.cpu().numpy()

    A, x = rng.uniform(0.5, 1, (M, K)).astype(dt), rng.uniform(0.5, 1, K).astype(dt)
    plain = run(A, x)
    # Inf in x: every row has the term, so all are Inf and none is NaN
    xi = x.copy()
    xi[K // 2] = np.inf
    np.testing.assert_array_equal(run(A, xi), np.full(M, np.inf, dt))
    # NaN and Inf in single elements of A: those rows alone
    B = A.copy()
    B[M // 2, K // 3], B[M - 1, K - 1] = np.nan, -np.inf
    got = run(B, x)
    other = np.ones(M, bool)
    other[[M // 2, M - 1]] = False
    assert np.isnan(got[M // 2]) and got[M - 1] == -np.inf
    np.testing.assert_array_equal(got[other], plain[other])

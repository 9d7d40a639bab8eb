"""GEMV at every alignment: leading dimensions of each residue, a matrix and
vectors off the 16-byte grid, extents at the edges of the row groups, row
blocks and column splits, on both kernels (row- and column-streaming)."""
import numpy as np
import pytest

from _tol import C_GEMM, eps

pytestmark = pytest.mark.gpu

# (rows, reduction): vectors' edges, one and several row groups / blocks,
# shared columns, splits (in clusters, and through scratch beyond 16)
SHAPES = [(1, 1), (3, 5), (31, 33), (124, 64), (125, 65), (128, 127), (129, 300), (257, 1023), (63, 9001),
          (5, 40003), (700, 2047), (9731, 67), (4999, 2049), (33000, 35)]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("cols_form", [False, True])
@pytest.mark.parametrize("M,K", SHAPES)
@pytest.mark.parametrize("off", [0, 1, 3])
def test_every_alignment(cuda, dt, cols_form, M, K, off):
    import gbblas
    torch = cuda
    rng = np.random.default_rng(M + 3 * K + off)
    A = rng.uniform(-1, 1, (M, K)).astype(dt)
    x, y0 = rng.uniform(-1, 1, K).astype(dt), rng.uniform(-1, 1, M).astype(dt)

    def dev(v, o):  # v on the device, `o` elements past a 16-byte boundary, guarded by NaN
        return torch.from_numpy(np.concatenate([np.full(o, np.nan, dt), v.ravel(), np.full(5, np.nan, dt)])).cuda()

    ta, tx, ty = dev(A.T if cols_form else A, off), dev(x, off // 2), dev(y0, 0)
    size = np.dtype(dt).itemsize
    # (matrix rows M x K row-major, or the same stored column-major)
    for _ in range(2):
        ty = dev(y0, 0)
        gbblas.call(f"gbblas_{'s' if dt == np.float32 else 'd'}gemv", 0 if cols_form else 1, 0, M, K,
                    ta.data_ptr() + off * size, tx.data_ptr() + off // 2 * size, 1, ty.data_ptr(), None)
        got = ty.cpu().numpy()
        assert np.all(np.isnan(got[M:]))
        exact = A.astype(np.longdouble) @ x + y0
        scale = np.abs(A).astype(np.float64) @ np.abs(x) + np.abs(y0)
        assert np.all(np.abs(got[:M] - exact) <= C_GEMM * max(K, 1) * eps(dt) * scale)
        if _ == 0:
            first = got
    np.testing.assert_array_equal(first, got)

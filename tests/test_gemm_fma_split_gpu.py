"""The register-tiled FMA GEMM: every fetch form (16-byte vectors, elements
along M / N, elements along K, general strides) and layout at the edges of its
tiles gives one set of bits, and with K cut over the CTAs of a cluster
(GBBLAS_FMA_TILE=5 / 6; double: by its own rule) results stay inside the
K-term bound and repeat."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64 = 5


def matrix(torch, X, layout, pad, step=1):
    """X on the device: row- (1) or column-major (0), rows `pad` elements
    longer than they need be, neighbours `step` apart; the strides."""
    v = X if layout else X.T
    pitch = v.shape[1] * step + pad
    buf = np.full((v.shape[0], pitch), -5, X.dtype)
    buf[:, :v.shape[1] * step:step] = v
    t = torch.from_numpy(buf).cuda()
    return t, ((pitch, step) if layout else (step, pitch))


def gemm(torch, A, B, C0, la, lb, lc, pad=0, step=1):
    import gbblas
    M, K = A.shape
    N = B.shape[1]
    a, sa = matrix(torch, A, la, pad, step)
    b, sb = matrix(torch, B, lb, pad, step)
    c, sc = matrix(torch, C0, lc, pad)
    args = (M, N, K, a.data_ptr(), *sa, b.data_ptr(), *sb, c.data_ptr(), *sc)
    if A.dtype == np.float32:
        gbblas.call("gbblas_sgemm", *args, 0, None)
    else:
        gbblas.call("gbblas_dgemm_ex", *args, FP64, None)
    gbblas.call("gbblas_check_stream", None)
    out = c.cpu().numpy()
    assert np.all(out[:, (N if lc else M):] == -5), "memory beside C changed"
    got = out[:, :N] if lc else out[:, :M].T
    return got


def operands(M, N, K, dtype, seed):
    rng = np.random.default_rng(seed)
    return tuple(rng.uniform(-1, 1, s).astype(dtype) for s in ((M, K), (K, N), (M, N)))


# around the 64 / 128 tiles and the 16-deep slices, down to one element
SHAPES = [(1, 1, 1), (63, 65, 15), (64, 64, 16), (65, 63, 17), (128, 129, 33), (130, 127, 64), (211, 190, 173)]


@pytest.mark.parametrize("tile", [0, 1])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_forms_and_layouts_same_bits(cuda, monkeypatch, tile, M, N, K):
    monkeypatch.setenv("GBBLAS_FMA_TILE", str(tile))
    A, B, C0 = operands(M, N, K, np.float32, M + N + K)
    want = gemm(cuda, A, B, C0, 1, 1, 1)
    for la, lb, lc in [(0, 0, 0), (0, 1, 0), (1, 0, 1), (0, 0, 1), (1, 1, 0)]:
        for pad, step in [(0, 1), (1, 1), (4, 1), (0, 2)]:
            np.testing.assert_array_equal(gemm(cuda, A, B, C0, la, lb, lc, pad, step), want)


# parts: 8, fewer by K, fewer by the tile count, one
@pytest.mark.parametrize("dtype,tile", [(np.float32, 5), (np.float32, 6), (np.float64, 0)])
@pytest.mark.parametrize("M,N,K", SHAPES + [(37, 70, 5000), (100, 300, 257), (700, 1000, 129), (1500, 1300, 40)])
def test_split_within_bound_and_repeats(cuda, monkeypatch, dtype, tile, M, N, K):
    monkeypatch.setenv("GBBLAS_FMA_TILE", str(tile))
    A, B, C0 = operands(M, N, K, dtype, M * 3 + N + K)
    big = np.longdouble if dtype == np.float64 else np.float64
    exact = A.astype(big) @ B.astype(big) + C0
    # a K-term sum in any order, plus the addition into C
    tol = (K + 2) * np.finfo(dtype).eps * (np.abs(A).astype(np.float64) @ np.abs(B) + np.abs(C0))
    for la, lb, lc in [(1, 1, 1), (0, 1, 0), (1, 0, 0)]:
        got = gemm(cuda, A, B, C0, la, lb, lc, 1)
        assert np.all(np.abs(got - exact) <= tol)
        np.testing.assert_array_equal(gemm(cuda, A, B, C0, la, lb, lc, 1), got)


def test_split_stays_within_the_servers_cta_cap(cuda, monkeypatch):
    """A heavy request capped to one CTA takes its tiles whole: the unsplit
    form's bits, not those of K cut over a cluster of eight."""
    import gbblas
    A, B, C0 = operands(37, 70, 5000, np.float32, 5)
    monkeypatch.setenv("GBBLAS_FMA_TILE", "0")
    whole = gemm(cuda, A, B, C0, 1, 1, 1)
    monkeypatch.setenv("GBBLAS_FMA_TILE", "5")
    assert not np.array_equal(gemm(cuda, A, B, C0, 1, 1, 1), whole)
    monkeypatch.delenv("GBBLAS_FMA_TILE")
    a, b, c = (cuda.from_numpy(x.copy()).cuda() for x in (A, B, C0))
    srv = gbblas.Server(streams=1, heavy_us=1, heavy_sm_percent=1, slice_us=-1)
    srv.wait(srv.submit(gbblas.Request(gbblas.OP_MTM, gbblas.F32, gbblas.ACCURACY_FP32, gbblas.LAST_ORDER, 37, 70, 5000,
                                       a.data_ptr(), b.data_ptr(), c.data_ptr())))
    srv.close()
    np.testing.assert_array_equal(c.cpu().numpy(), whole)


@pytest.mark.parametrize("la,lb,lc", [(1, 1, 1), (0, 1, 0), (1, 0, 1)])
@pytest.mark.parametrize("K", [1, 2, 7, 15, 16, 17, 31, 33])
def test_double_adds_nothing_beyond_k(cuda, K, la, lb, lc):
    """Products that underflow to -0 into a C of -0: every sum is -0, unless a
    k that does not exist adds its +0 (and takes the time of one that does)."""
    A, B = np.full((70, K), -1e-200), np.full((K, 67), 1e-200)
    got = gemm(cuda, A, B, np.full((70, 67), -0.0), la, lb, lc, 1)
    assert np.all(got == 0) and np.all(np.signbit(got))

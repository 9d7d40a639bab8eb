"""AUTO's guard over the double digit GEMM samples a quarter of K, or all of it
in tiles whose operands are too thin for that.  The choice is a tile's own:
rows elsewhere, and rows whose blocks the guard rejects however much is sampled
(zero, Inf, NaN), leave a tile's bits as they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AUTO = 3


def product(torch, A, B):
    import gbblas
    C = torch.full((A.shape[0], B.shape[1]), 0.25, dtype=torch.float64, device="cuda")
    gbblas.gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C, accuracy=AUTO)
    gbblas.call("gbblas_check_stream", None)
    return C.cpu().numpy()


def turns_on_the_choice(M, N, K, rng):
    """Rows and columns that are never large at the same k among the 32 of every
    128 that the quarter takes, and are elsewhere: their sampled sums call for
    the quarter, which rejects every block; all of K would accept them."""
    A, B = rng.uniform(-1, 1, (M, K)), rng.uniform(-1, 1, (K, N))
    k = np.arange(K)
    A[:, (k % 128 < 32) & (k % 32 >= 16)] *= 2.0 ** -20
    B[(k % 128 < 32) & (k % 32 < 16), :] *= 2.0 ** -20
    return A, B


@pytest.mark.parametrize("row", [200, 60])  # in the other tile, in the tile itself
@pytest.mark.parametrize("poke", ["zero", "inf", "nan", "thin"])
def test_a_tile_decides_for_itself(cuda, row, poke):
    M, N, K = 256, 32, 1024
    A, B = turns_on_the_choice(M, N, K, np.random.default_rng(row))
    plain = product(cuda, A, B)
    if poke == "zero":
        A[row] = 0.0
    elif poke == "thin":
        A[row] *= 2.0 ** -20
        A[row, 0] = 1.0
    else:
        A[row, 5] = np.inf if poke == "inf" else np.nan
    got = product(cuda, A, B)
    # (a thin row's own tile takes all of K: other bits, inside the bound)
    same = np.arange(M) < 128 if poke == "thin" and row >= 128 else np.arange(M) != row
    if not (poke == "thin" and row < 128):
        np.testing.assert_array_equal(got[same], plain[same])
    if poke in ("inf", "nan"):
        assert np.all(~np.isfinite(got[row]))
    finite = np.arange(M) != row if poke in ("inf", "nan") else np.ones(M, bool)
    exact = A[finite].astype(np.longdouble) @ B.astype(np.longdouble) + 0.25
    bound = 2 * K * 2.0 ** -52 * (np.abs(A[finite]) @ np.abs(B) + 0.25)
    assert np.all(np.abs(got[finite] - exact) <= bound)


# several tiles per CTA, whole ones and (K of five chunks) cut ones, the choice
# changing from one to the next; K of one chunk and a stage
@pytest.mark.parametrize("M,N,K", [(128 * 17, 320, 600), (128 * 20 + 5, 310, 130)])
def test_choices_mixed_over_tiles(cuda, M, N, K):
    rng = np.random.default_rng(M + K)
    A, B = rng.uniform(-1, 1, (M, K)), rng.uniform(-1, 1, (K, N))
    wide = (np.arange(M) // 128) % 2 == 1
    A[wide] *= np.exp2(rng.integers(-10, 11, (int(wide.sum()), K)))
    A[wide & (np.arange(M) % 128 == 77)] = 0.0
    B[:, 64:96] *= np.exp2(rng.integers(-10, 11, (K, 32)))
    got = product(cuda, A, B)
    exact = A.astype(np.longdouble) @ B.astype(np.longdouble) + 0.25
    assert np.all(np.abs(got - exact) <= 2 * K * 2.0 ** -52 * (np.abs(A) @ np.abs(B) + 0.25))
    np.testing.assert_array_equal(product(cuda, A, B), got)


def test_the_quarter_where_its_sums_vary_little(cuda):
    """Sums whose smallest product is three times the limit and varies by a
    twentieth: the quarter is taken.  Shown on operands built so that it rejects
    every block (never large at the same sampled k), which are then sums of
    fused multiply-adds in order of k, as the pipes add them."""
    from fractions import Fraction
    M, N, K = 128, 32, 16384
    A, B = turns_on_the_choice(M, N, K, np.random.default_rng(3))
    A, B = A / 8, B / 8
    A[:, 100], B[101, :] = 0.75, 0.75  # (not sampled) the rows' and columns' largest, digits of 96
    got = product(cuda, A, B)
    for i, j in ((0, 0), (77, 13), (127, 31)):
        s = 0.0
        for x, y in zip(A[i].tolist(), B[:, j].tolist()):
            s = float(Fraction(x) * Fraction(y) + Fraction(s))
        assert got[i, j] == s + 0.25

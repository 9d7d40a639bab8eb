"""Padding rows that hold another call's NaN (test_gemm_tc_padding_gpu), in the
forms a single call of a tile or two does not take: a group, CTA pairs, K cut
into parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BF16X3, BF16X6 = 1, 4
SHAPES = [(1, 1, 64), (257, 129, 100), (100, 200, 520), (300, 40, 1000)]


@pytest.mark.parametrize("acc", [BF16X3, BF16X6])
@pytest.mark.parametrize("form", ["group", "pairs", "split"])
@pytest.mark.parametrize("layout", [0, 1])
def test_stale_nan_in_padding_rows(cuda, monkeypatch, acc, form, layout):
    import gbblas
    torch = cuda
    if form != "group":
        monkeypatch.setenv("GBBLAS_TC_PAIR" if form == "pairs" else "GBBLAS_TC_SPLITK", "1" if form == "pairs" else "3")
    rng = np.random.default_rng(acc + layout)
    dev = lambda X: torch.from_numpy(np.ascontiguousarray(X if layout else X.T)).cuda()  # noqa: E731
    view = lambda t: t if layout else t.t()  # noqa: E731
    ops = []
    for M, N, K in SHAPES:
        A, B = rng.integers(-8, 9, (M, K)).astype(np.float32), rng.integers(-8, 9, (K, N)).astype(np.float32)
        C = rng.integers(-50, 51, (M, N)).astype(np.float32)
        ops.append((view(dev(A)), view(dev(B)), torch.from_numpy(C).cuda(), A.astype(np.float64) @ B + C))
    bad = torch.full((2048, 2048), float("nan"), device="cuda")

    def stale():
        gbblas.gemm(bad, bad, torch.zeros(2048, 2048, device="cuda"), accuracy=acc)

    if form == "group":
        stale()
        gbblas.gemm_grouped([gbblas.gemm_desc(a, b, c) for a, b, c, _ in ops], accuracy=acc)
    else:
        for a, b, c, _ in ops:
            stale()
            gbblas.gemm(a, b, c, accuracy=acc)
    gbblas.call("gbblas_check_stream", None)
    for _, _, c, want in ops:
        np.testing.assert_array_equal(c.cpu().numpy(), want)

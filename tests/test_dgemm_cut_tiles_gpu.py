"""Double GEMM on the tensor-core digits: tiles of the last, incomplete round
are cut along K and their integer sums added from slots.  The same rows and
columns inside a product whose tiles fill whole rounds (128 x 152 rows by 32
columns: one tile per SM) are computed whole, so the bits must agree; AUTO's
guard must decide the same too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AUTO, DIGITS7, DIGITS8 = 3, 6, 7


def product(torch, A, B, acc):
    import gbblas
    C = torch.full((A.shape[0], B.shape[1]), 0.25, dtype=torch.float64, device="cuda")
    gbblas.gemm(A, B, C, accuracy=acc)
    gbblas.call("gbblas_check_stream", None)
    return C


# one row block to several; K from two parts to one per CTA, chunks and stages left over
@pytest.mark.parametrize("acc", [DIGITS7, DIGITS8, AUTO])
@pytest.mark.parametrize("M,N,K", [(128, 32, 513), (100, 20, 1000), (128, 32, 4096), (300, 70, 2217), (128, 32, 40001)])
@pytest.mark.parametrize("wide", [False, True])
def test_cut_tiles_same_bits_as_whole(cuda, acc, M, N, K, wide):
    torch = cuda
    rng = np.random.default_rng(M + K + wide)

    def values(shape):
        v = rng.uniform(-1, 1, shape)
        return torch.from_numpy(v * np.exp2(rng.integers(-10, 11, shape)) if wide else v).cuda()

    A, B = values((M, K)), values((K, N))
    cut = product(torch, A, B, acc)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    whole = torch.empty_like(cut)
    for n in range(0, N, 32):  # 32 columns at a time, rows padded to one tile per SM
        cols = B[:, n:n + 32].contiguous()
        tall = torch.cat([A, A.new_ones(128 * sms - M, K)])
        whole[:, n:n + 32] = product(torch, tall, cols, acc)[:M]
    assert torch.equal(cut, whole)
    exact = (A.cpu().numpy().astype(np.longdouble) @ B.cpu().numpy().astype(np.longdouble)) + 0.25
    mag = (A.abs() @ B.abs()).cpu().numpy()
    rows, cols = A.abs().amax(1).cpu().numpy(), B.abs().amax(0).cpu().numpy()
    # AUTO: the pipes' bound; the digits: theirs, on the rows' and columns' largest (scales up to twice those)
    bound = 2 * K * 2.0 ** -52 * (mag + 0.25)
    if acc != AUTO:
        bound = bound + 9 * 2.0 ** -56 * K * 4 * np.outer(rows, cols)
    assert np.all(np.abs(cut.cpu().numpy() - exact) <= bound)

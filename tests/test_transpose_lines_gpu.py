"""Transposes large enough to be written in whole lines (200 MB moved, C's rows
off the 128-byte lines): every layout pair, padded and offset C, extents that
leave partial strips, chunks and column blocks.  Copies, so bit for bit."""
import pytest

pytestmark = pytest.mark.gpu

# (M, N, C's extra pitch, C's offset in elements)
CASES = [(5003, 5009, 0, 0), (40001, 641, 0, 0), (127, 200003, 3, 1), (8192, 4000, 1, 0), (8192, 3200, 0, 5),
         (63, 400007, 0, 0)]


@pytest.mark.parametrize("dt", ["s", "d"])
@pytest.mark.parametrize("la", [0, 1])
@pytest.mark.parametrize("lc", [0, 1])
@pytest.mark.parametrize("M,N,pad,off", CASES)
def test_lines(cuda, dt, la, lc, M, N, pad, off):
    import gbblas
    torch = cuda
    T = torch.float32 if dt == "s" else torch.float64
    # (values are bit patterns of a counter: every element differs)
    A = torch.arange(M * N, device="cuda", dtype=torch.int32 if dt == "s" else torch.int64).view(T)
    A = A.view(M, N) if la else A.view(N, M).t()
    pitch = (M if lc else N) + pad
    buf = torch.full((off + (N if lc else M) * pitch + 9,), -3.0, device="cuda", dtype=T)
    C = buf[off:off + (N if lc else M) * pitch].view(-1, pitch)
    rsc, csc = (pitch, 1) if lc else (1, pitch)
    gbblas.call(f"gbblas_{dt}transpose", M, N, A.data_ptr(), A.stride(0), A.stride(1), C.data_ptr(), rsc, csc, None)
    I = torch.int32 if dt == "s" else torch.int64
    got, want = (C[:, :M], A.t()) if lc else (C[:, :N], A)
    assert torch.equal(got.contiguous().view(I), want.contiguous().view(I))
    # C^T's other half: nothing beside C changed
    assert bool((C[:, (M if lc else N):] == -3.0).all()) and bool((buf[:off] == -3.0).all()) and bool((buf[-9:] == -3.0).all())


def test_no_exchange_is_no_slower_than_one(cuda):
    """A and C contiguous along the same index: a copy, without an exchange
    through shared memory and so not slower than the transpose of that size."""
    import gbblas
    torch = cuda
    M, N = 9001, 7003
    A, C, flush = (torch.rand(n, device="cuda") for n in (M * N, M * N, 64 << 20))

    def best(rsc, csc):
        times = []
        for _ in range(15):
            flush.fill_(1.0)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            gbblas.call("gbblas_stranspose", M, N, A.data_ptr(), N, 1, C.data_ptr(), rsc, csc, None)
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    assert best(1, N) <= best(M, 1)

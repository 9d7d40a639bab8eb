"""AUTO's fix-up of the rows its guard rejects is shared out over the SMs: one
such row beside a product that fills them must not multiply its time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def best_ms(torch, call):
    for _ in range(3):
        call()
    times = []
    for _ in range(20):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(5):
            call()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) / 5)
    return min(times)


# outputs beyond, at and around one share; a row of A, a column of B, both
@pytest.mark.parametrize("where", ["a", "b", "ab"])
@pytest.mark.parametrize("M,N", [(1158, 4096), (63, 129), (64, 64), (200, 65)])
def test_rejected_rows(cuda, monkeypatch, where, M, N):
    import gbblas
    torch = cuda
    monkeypatch.setenv("GBBLAS_GEMM_AUTO", "1")
    rng = np.random.default_rng(M + N)
    K = 201
    A, B = (np.sign(rng.uniform(-1, 1, s)) * rng.uniform(0.5, 1, s) for s in ((M, K), (K, N)))
    a, b = (torch.from_numpy(x.astype(np.float32)).cuda() for x in (A, B))
    c = torch.zeros(M, N, device="cuda")
    call = lambda: gbblas.gemm(a, b, c, accuracy=gbblas.ACCURACY_AUTO)  # noqa: E731
    plain = best_ms(torch, call)
    # an element further below its row's largest than K = 201 allows
    if "a" in where:
        a[M // 2, 7] = 2.0 ** -30
    if "b" in where:
        b[9, N - 1] = 2.0 ** -30
    c.zero_()
    call()
    got = c.cpu().numpy()
    A, B = a.double().cpu().numpy(), b.double().cpu().numpy()
    assert np.all(np.abs(got - A @ B) <= 2 * K * 2.0 ** -23 * (np.abs(A) @ np.abs(B)))
    if M * N > 1000000:
        assert best_ms(torch, call) < 2 * plain

"""Admission of double GEMMs on tensor-core digits: a request needs its
operands, scales, digit planes and fix-up list, no more; what only makes it
faster (slots for cutting its last tiles along K, the guard's sampled sums) is
taken where the budget has it.  The bits do not depend on the cut."""
import numpy as np
import pytest

from test_serve_gpu import AUTO, ReqCase

pytestmark = pytest.mark.gpu

DIGITS7, DIGITS8 = 6, 7


def needed(M, N, K, accuracy):
    up = lambda v, m: (v + m - 1) // m * m  # noqa: E731
    mp, np_, kp = up(M, 128), up(N, 32), up(K, 32)
    planes = 7 if accuracy == DIGITS7 else 8  # AUTO: seven digits and the guard
    tiles = (mp // 128) * (np_ // 32)
    scratch = 256 + up(4 * mp, 256) + up(4 * np_, 256) + up(2 * planes * mp * kp, 256) + up(2 * planes * np_ * kp, 256)
    if accuracy == AUTO:
        scratch += up(4 * (1 + 8 * tiles), 256)
    return 8 * (M * K + K * N + M * N) + scratch


# 64 tiles in two parts, 12 tiles in four, K too short for a cut; heavy ones
# with and without slices
@pytest.mark.parametrize("accuracy", [AUTO, DIGITS7, DIGITS8])
@pytest.mark.parametrize("dims", [(512, 512, 512), (300, 100, 1100), (512, 512, 100)])
@pytest.mark.parametrize("heavy", [{}, {"heavy_us": 20}, {"heavy_us": 20, "slice_us": -1}])
def test_admitted_with_what_it_needs(cuda, accuracy, dims, heavy):
    import gbblas
    torch = cuda
    least = needed(*dims, accuracy)
    c = ReqCase(torch, np.random.default_rng(dims[2]), gbblas.OP_MTM, gbblas.F64, 1, dims, accuracy)
    outs = []
    for budget in (least, least + (1 << 20), 1 << 30):
        srv = gbblas.Server(streams=2, budget_bytes=budget, **heavy)
        srv.wait(srv.submit(c.request()))
        assert srv.stats()["peak_inflight_bytes"] <= budget
        srv.close()
        outs.append(c.outs[-1])
        if accuracy == AUTO:
            c.check(outs[-1])
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    srv = gbblas.Server(streams=2, budget_bytes=least - 1, **heavy)
    with pytest.raises(gbblas.GbblasError) as e:
        srv.submit(c.request())
    assert e.value.status == 3  # GBBLAS_STATUS_ALLOC_FAILED
    srv.close()

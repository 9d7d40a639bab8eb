"""dot at the edges of its launch forms (one CTA, one cluster, the grid with
partials) and where a warp's totals leave the range FP32 pairs can hold."""
import numpy as np
import pytest

from oracle import oracle as O

from _tol import C_KAHAN, eps
from test_dot_gpu import gpu_dot

pytestmark = pytest.mark.gpu

# one CTA up to 8192 (f32) / 2048 (f64) elements, one cluster up to eight
# times that, partials beyond; 4-element vectors and their remainders
EDGES = [31, 2047, 2048, 2049, 8191, 8192, 8193, 16384, 16387, 40000, 65535, 65536, 65537, 300001]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("offset", [0, 1])
def test_launch_forms(cuda, dt, n, offset):
    rng = np.random.default_rng(n + offset)
    a, b = rng.uniform(-1, 1, n).astype(dt), rng.uniform(-1, 1, n).astype(dt)
    got = gpu_dot(cuda, a, b, offset=offset)
    exact, absdot = O.dot_exact(a, b)
    bound = (C_KAHAN if dt == np.float32 else 2 * np.sqrt(n)) * eps(dt) * absdot + eps(dt) * abs(exact)
    assert abs(got - exact) <= bound
    assert gpu_dot(cuda, a, b, offset=offset) == got


@pytest.mark.parametrize("n", [2048])
def test_totals_beyond_float_range(cuda, n):
    """Threads' sums of 3e38 and -3e38 (4 consecutive elements each): a warp's
    running total passes FLT_MAX, the dot does not."""
    a = np.where(np.arange(n) // 64 % 2 == 0, np.float32(3e38), np.float32(-3e38)).astype(np.float32)
    a[n // 128 * 128:] = 0.0
    a[-1] = 2.0 ** 100
    b = np.ones(n, np.float32)
    # 3e38 and -3e38 cancel exactly, but for one whose place the 2^100 takes
    # where n is a multiple of 128; what is left beside them in a lane, and the
    # result, are rounded at their size, at most half an ulp of 3e38
    assert abs(gpu_dot(cuda, a, b) - a.astype(np.longdouble).sum()) <= 2.0 ** 103
    small = (a * np.float32(2.0 ** -30)).astype(np.float32)
    small[-1] = 0.0
    assert gpu_dot(cuda, small, b) == small.astype(np.longdouble).sum()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("n", [100, 20000, 200000])
def test_not_finite_stays_not_finite(cuda, bad, n):
    a, b = np.ones(n, np.float32), np.ones(n, np.float32)
    a[n // 3] = bad
    assert not np.isfinite(gpu_dot(cuda, a, b))
    assert not np.isfinite(gpu_dot(cuda, a.astype(np.float64), b.astype(np.float64)))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [0, 1] + EDGES + [2500000, 2600001])  # (... and the full grid, in clusters)
def test_allocation_free_form_gives_the_same_bits(cuda, n, offset):
    import gbblas
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.rand(n + offset, generator=g, device="cuda") * 2 - 1 for _ in range(2))
    out = torch.full((2,), 7.0, device="cuda")
    for i, fn in enumerate(("gbblas_sdot", "gbblas_sdot_noalloc")):
        gbblas.call(fn, n, a[offset:].data_ptr(), b[offset:].data_ptr(), out[i:].data_ptr(), None)
    torch.cuda.synchronize()
    assert out[0].item() == out[1].item()

"""CSR SpMV by row blocks with given lanes and unroll: row lengths at the edges
of one and two passes, and the compensated f32 sums beyond one pass."""
import numpy as np
import pytest

from sciwasm.sparse_b200 import _lib

pytestmark = pytest.mark.gpu


def _cancelling(lens, dt, seed):
    """Rows whose products are exact in dt and cancel: +-2^20 in pairs with
    values of order 1 between them."""
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    N, nnz = len(lens), int(rp[-1])
    col = rng.integers(0, N, nnz).astype(np.int32)
    p = rng.integers(-2048, 2048, nnz) / 1024.0
    for s, e in zip(rp[:-1], rp[1:]):
        k = (e - s) // 4 * 2
        big = rng.choice(np.arange(s, e), k, replace=False)
        p[big[0::2]] += 1 << 20  # in [2^20 - 2, 2^20 + 2): cut to 24 bits below
        p[big[1::2]] -= 1 << 20
    p = np.float32(p).astype(dt)
    x = (2.0 ** rng.integers(-3, 4, N)).astype(dt)
    return rp, col, (p / x[col]).astype(dt), x


@pytest.mark.parametrize("grid", [0, 1])
@pytest.mark.parametrize("unroll", [2, 4, 8])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_edges_of_passes(gpu, dt, lanes, unroll, grid):
    short = lanes * unroll
    edges = [0, 1, 2, lanes, short - 1, short, short + 1, short + short // 2, 2 * short - 1,
             2 * short, 2 * short + 1, 3 * short + 5]
    rng = np.random.default_rng(lanes * unroll)
    lens = np.concatenate([rng.choice(edges, 3 * len(edges)), edges, [short + 1] * 32, [short] * 40])
    rp, col, val, x = _cancelling(lens, dt, 3)
    N = lens.size
    A = gpu.csr_from_host(rp, col, val)
    A.opts = _lib.CsrOpts(0, lanes, unroll, grid)
    yv = gpu.create_vec(N, 0, dt)
    gpu.spmv(A, gpu.vec_from_host(x), yv)
    y = yv.array().astype(np.float64)
    u = np.finfo(dt).eps / 2
    for i in range(N):
        p = val[rp[i]:rp[i + 1]].astype(np.float64) * x[col[rp[i]:rp[i + 1]]]
        want, mass, n = p.sum(), np.abs(p).sum(), len(p)
        # products and the 64-bit sums are exact.  A plain sum of n terms is off by
        # n u sum|p| at most, a compensated one by u |sum| and n^2 u^2 sum|p|
        # (the lanes' sums are compensated again when they are added)
        if dt == np.float32 and n > short:
            tol = 2 * u * abs(want) + 4 * n * n * u * u * mass
        else:
            tol = n * u * mass
        assert abs(y[i] - want) <= tol, (i, n, y[i], want, tol)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["five", "boundary", "eleven", "poisson4", "poisson10", "mixed4",
                                  "mixed10", "empty"])
def test_default_sums_of_short_rows(gpu, dt, kind):
    """Without options, rows of up to one pass are summed as two lanes (four for
    means above 6) with four entries each sum them, bit for bit."""
    rng = np.random.default_rng(5)
    N = 32 * 70 + 13
    lens = {"five": np.full(N, 5), "boundary": np.where(np.arange(N) % 37, 7, 6),
            "eleven": np.full(N, 11), "poisson4": rng.poisson(4, N), "poisson10": rng.poisson(10, N),
            "mixed4": np.where(np.arange(N) // 32 % 2, 4, rng.poisson(4, N)),
            "mixed10": np.where(np.arange(N) // 32 % 2, 9, rng.poisson(10, N)),
            "empty": np.where(rng.random(N) < 0.9, 0, 8)}[kind]
    lanes = 2 if lens.mean() <= 6 else 4
    if dt == np.float64:
        lens = np.minimum(lens, 4 * lanes)  # (four lanes take two passes in FP64)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, N, rp[-1]).astype(np.int32)
    A = gpu.csr_from_host(rp, col, rng.standard_normal(rp[-1]).astype(dt))
    x, y0 = gpu.vec_from_host(rng.standard_normal(N).astype(dt)), rng.standard_normal(N).astype(dt)
    ys = []
    for opts in (None, _lib.CsrOpts(0, lanes, 4, 0)):
        A.opts = opts
        yv = gpu.vec_from_host(y0)
        gpu.spmv(A, x, yv)
        ys.append(yv.array())
    assert np.array_equal(ys[0].view(np.uint8), ys[1].view(np.uint8))

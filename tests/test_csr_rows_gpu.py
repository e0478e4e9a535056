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

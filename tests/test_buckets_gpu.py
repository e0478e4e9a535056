"""The bucket sort of coo_csr and of the CSR transpose, bit for bit against the
oracle, at the edges of its parts: rows on both sides of the rank, small, medium
and large sorts, buckets that have to be cut down, a row beyond them (radix
sort), repeated coordinates, empty rows and one-row matrices, neighbours in one
bucket, indices out of range found after the prefix that is checked first."""
import numpy as np
import pytest

from sciwasm.sparse_b200 import SparseError

pytestmark = pytest.mark.gpu


def _ub(a):
    return np.ascontiguousarray(a).view(np.uint8)


def _coo(lens, N, seed, dup=0.0, order="shuffled"):
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens, np.int64)
    row = np.repeat(np.arange(lens.size), lens)
    col = rng.integers(0, N, row.size)
    if dup:  # many equal (row, col) pairs: their order is the input's
        col = np.where(rng.random(row.size) < dup, col % 3, col)
    p = {"shuffled": lambda: rng.permutation(row.size),
         "rows": lambda: np.arange(row.size),              # rows in order, columns not
         "cols": lambda: np.lexsort((row, col)),
         "reversed": lambda: np.arange(row.size)[::-1]}[order]()
    return row[p].astype(np.int32), col[p].astype(np.int32), rng.uniform(-1, 1, row.size)


def _lens(kind):
    rng = np.random.default_rng(1)
    if kind == "ranks":      # one bucket holds rows of 255, 256, 257 and short ones
        return np.concatenate([[255, 256, 257, 0, 1, 2], rng.integers(0, 9, 3000)])
    if kind == "small":      # buckets at 1023, 1024 and 1025 entries
        return np.concatenate([np.full(341, 3), [1, 1024 - 3], np.full(900, 3)])
    if kind == "large":      # rows of 2047, 2048, 2049 and 8192 entries
        return np.concatenate([[2047, 2048, 2049, 8192], rng.integers(0, 5, 2000)])
    if kind == "cut":        # long rows next to one another among short ones
        return np.concatenate([np.full(40, 1500), rng.integers(0, 4, 60_000)])
    if kind == "radix":      # a row beyond a bucket
        return np.concatenate([[9000], rng.integers(0, 4, 5000)])
    if kind == "empty":      # most rows empty, the last ones too
        n = np.zeros(100_000, np.int64)
        n[rng.integers(0, 70_000, 900)] = 2
        return n
    if kind == "one":
        return np.array([700])
    return rng.integers(9, 13, 20_000)  # "even"


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind,dup,order", [
    ("ranks", 0.3, "shuffled"), ("small", 0.0, "shuffled"), ("large", 0.5, "shuffled"),
    ("cut", 0.2, "shuffled"), ("radix", 0.2, "shuffled"), ("empty", 0.0, "shuffled"),
    ("one", 0.5, "shuffled"), ("even", 0.1, "rows"), ("even", 0.1, "cols"),
    ("even", 0.0, "reversed"), ("even", 0.9, "shuffled")])
def test_coo_csr_buckets(gpu, oracle, dt, kind, dup, order):
    lens = _lens(kind)
    N = lens.size
    row, col, val = _coo(lens, N, 3, dup, order)
    val = val.astype(dt)
    want = oracle.coo_csr(row, col, val, N)
    A = gpu.coo_csr(gpu.coo_from_host(row, col, val, N))
    for got, w in zip((A.row_array(), A.col_array(), A.val_array()), want):
        assert np.array_equal(_ub(got), _ub(w)), kind


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["ranks", "large", "cut", "empty", "one", "even"])
def test_transpose_csr_buckets(gpu, oracle, dt, kind):
    """Columns of the lengths that the rows above have (skewed columns)."""
    lens = _lens(kind)
    N = lens.size
    col, row, val = _coo(lens, N, 5, 0.2)
    rp, c, v = oracle.coo_csr(row, col, val.astype(dt), N)
    B = gpu.transpose(gpu.csr_from_host(rp, c, v))
    want = oracle.transpose_csr(rp, c, v)
    for got, w in zip((B.row_array(), B.col_array(), B.val_array()), want):
        assert np.array_equal(_ub(got), _ub(w)), kind


@pytest.mark.parametrize("where", ["row", "col", "negative"])
def test_index_out_of_range_after_the_prefix(gpu, where):
    row, col, val = _coo(np.full(30_000, 4), 30_000, 9)
    A = gpu.coo_from_host(row, col, val, 30_000)
    bad = {"row": (row, 30_000), "col": (col, 30_000), "negative": (col, -1)}[where]
    bad[0][100_000] = bad[1]
    A.row_index.upload(row)
    A.col_index.upload(col)
    with pytest.raises(SparseError):
        gpu.coo_csr(A)


def _long(kind):
    rng = np.random.default_rng(2)
    if kind == "radix":     # one row beyond a bucket, found by the count
        return _lens("radix")
    if kind == "hub":       # found by the sample before it
        return np.concatenate([rng.integers(0, 12, 150_000), [120_000], rng.integers(0, 12, 50_000)])
    if kind == "hubs":      # missed or met by the sample, as it falls
        return np.concatenate([rng.integers(0, 12, 100_000), np.full(5, 13_000),
                               rng.integers(0, 12, 100_000)])
    # a bucket that has to be cut down to rows of their own
    return np.concatenate([rng.integers(0, 3, 40_000), np.full(9, 8192), rng.integers(0, 3, 9_000)])


def _sorted(row, col, val, N):
    """The stable sort by (row, col) that coo_csr is (the oracle's bubble sort
    takes minutes on rows of this length)."""
    p = np.lexsort((col, row))
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=N))]).astype(np.int32)
    return rp, col[p], val[p]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["radix", "hub", "hubs", "own"])
def test_rows_beyond_buckets(gpu, dt, kind):
    """coo_csr with such rows, and the transpose with such columns."""
    lens = _long(kind)
    N = lens.size
    row, col, val = _coo(lens, N, 7, 0.2)
    val = val.astype(dt)
    A = gpu.coo_csr(gpu.coo_from_host(row, col, val, N))
    for got, w in zip((A.row_array(), A.col_array(), A.val_array()), _sorted(row, col, val, N)):
        assert np.array_equal(_ub(got), _ub(w)), kind
    rp, c, v = _sorted(col, row, val, N)
    B = gpu.transpose(gpu.csr_from_host(rp, c, v))
    at = np.repeat(np.arange(N, dtype=np.int32), np.diff(rp))
    for got, w in zip((B.row_array(), B.col_array(), B.val_array()), _sorted(c, at, v, N)):
        assert np.array_equal(_ub(got), _ub(w)), kind


@pytest.mark.parametrize("N,per_row", [(3, 500), (1000, 65), (9471, 9), (30_011, 20), (320_001, 3)])
def test_transpose_rows_per_warp(gpu, N, per_row):
    """One row to a warp up to 32, the last warp with fewer, empty rows between."""
    rng = np.random.default_rng(N)
    lens = np.where(rng.random(N) < 0.1, 0, rng.integers(0, 2 * per_row, N))
    row = np.repeat(np.arange(N, dtype=np.int32), lens)
    rp, c, v = _sorted(row, rng.integers(0, N, row.size).astype(np.int32),
                       rng.uniform(-1, 1, row.size), N)
    B = gpu.transpose(gpu.csr_from_host(rp, c, v))
    for got, w in zip((B.row_array(), B.col_array(), B.val_array()), _sorted(c, row, v, N)):
        assert np.array_equal(_ub(got), _ub(w))


@pytest.mark.parametrize("bad", [-1, 200_001, 2**31 - 1])
def test_index_out_of_range_beside_a_hub(gpu, bad):
    """The sample ends the count; the indices are checked all the same."""
    lens = _long("hub")
    N = lens.size
    row, col, val = _coo(lens, N, 9)
    A = gpu.coo_from_host(row, col, val, N)
    col[-1000] = bad
    A.col_index.upload(col)
    with pytest.raises(SparseError):
        gpu.coo_csr(A)

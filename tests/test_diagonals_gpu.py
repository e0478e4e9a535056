"""num_diags, csr_dia and csr_ell at the edges of their block's rows, staged
entries and known diagonals: few diagonals all seen in the first and last
rows, some only in the middle, 64 / 65 / many of them, rows that are unsorted
or repeat a column, and row pointers that do not ascend.  Bit-exact against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band(N, offsets, dt, keep=1.0, seed=0):
    rng = np.random.default_rng(seed + N)
    rows = np.repeat(np.arange(N, dtype=np.int64), len(offsets))
    col = rows + np.tile(np.asarray(offsets, np.int64), N)
    ok = (col >= 0) & (col < N) & (rng.random(col.size) < keep)
    rows, col = rows[ok], col[ok]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=N))]).astype(np.int32)
    return rp, col.astype(np.int32), rng.standard_normal(col.size).astype(dt)


def _check(gpu, oracle, rp, col, val, upload=None):
    A = gpu.csr_from_host(rp if upload is None else upload, col, val)
    A.row_index.upload(rp)
    want = oracle.csr_dia(rp, col, val)
    nd, stride = oracle.num_diags(rp, col)
    assert gpu.num_diags(A) == [nd, stride]
    D = gpu.csr_dia(A)
    assert (D is None) == (want is None)
    if want is not None:
        assert (D.ndiags, D.stride) == (want[2], want[3])
        assert np.array_equal(D.offset_array(), want[0])
        assert D.data_array().tobytes() == want[1].tobytes()
    want_ell = oracle.csr_ell(rp, col, val)
    E = gpu.csr_ell(A)
    assert (E is None) == (want_ell is None)
    if want_ell is not None:
        assert E.ncols == want_ell[2]
        assert np.array_equal(E.indices_array(), want_ell[0])
        assert E.data_array().tobytes() == want_ell[1].tobytes()
    return want is not None


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("N", [1, 2, 127, 128, 129, 1023, 1024, 1025, 2047, 2048, 2049, 5000])
def test_row_edges(gpu, oracle, N, dt):
    assert _check(gpu, oracle, *_band(N, [-3, 0, 1, 2], dt))
    assert _check(gpu, oracle, *_band(N, [-(N // 2), 0, N // 2] if N > 1 else [0], dt))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("width", [7, 8, 16, 27, 28, 32, 63, 64, 65, 130])
def test_widths(gpu, oracle, width, dt):
    offsets = list(range(-(width // 2), width - width // 2))
    assert _check(gpu, oracle, *_band(6000, offsets, dt))
    assert _check(gpu, oracle, *_band(6000, offsets, dt, keep=0.7))


@pytest.mark.parametrize("at", [1023, 1024, 3000, 4000 - 1025, 4000 - 1024])
@pytest.mark.parametrize("width", [5, 64])
def test_diagonal_of_one_row(gpu, oracle, at, width):
    offsets = list(range(-2, width - 2))
    rp, col, val = _band(4000, offsets, np.float64)
    col[rp[at + 1] - 1] = min(at + width + 40, 3999)
    assert _check(gpu, oracle, rp, col, val)


def test_all_in_the_middle_and_none(gpu, oracle):
    rp, col, val = _band(9000, [-1, 0, 1], np.float64)
    keep = np.zeros(9000, bool)
    keep[2000:7000] = True
    k = np.repeat(keep, np.diff(rp))
    rp = np.concatenate([[0], np.cumsum(np.diff(rp) * keep)]).astype(np.int32)
    assert _check(gpu, oracle, rp, col[k], val[k])


@pytest.mark.parametrize("width", [6, 70])
def test_unsorted_and_repeated(gpu, oracle, width):
    rp, col, val = _band(4100, list(range(-1, width - 1)), np.float32)
    rng = np.random.default_rng(1)
    for i in range(0, 4100, 7):
        col[rp[i]:rp[i + 1]] = rng.permutation(col[rp[i]:rp[i + 1]])
    for i in range(3, 4000, 11):
        col[rp[i] + 2] = col[rp[i] + rng.integers(0, 2)]
    assert _check(gpu, oracle, rp, col, val)


def test_dense_rows_of_many_diagonals(gpu, oracle):
    rng = np.random.default_rng(3)
    full = rng.random((300, 300)) < 0.7
    rp = np.concatenate([[0], np.cumsum(full.sum(1))]).astype(np.int32)
    col = np.nonzero(full)[1].astype(np.int32)
    assert _check(gpu, oracle, rp, col, rng.standard_normal(col.size).astype(np.float32))


@pytest.mark.parametrize("N", [33, 5000, 400_003])
def test_scattered_diagonals(gpu, oracle, N):
    rng = np.random.default_rng(N)
    lens = rng.integers(0, 9, N)
    lens[N // 2] = 3000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, N, rp[-1]).astype(np.int32)
    _check(gpu, oracle, rp, col, rng.standard_normal(col.size))


@pytest.mark.parametrize("width", [4, 70])
def test_row_pointers_that_do_not_ascend(gpu, oracle, width):
    rp, col, val = _band(3000, list(range(-1, width - 1)), np.float64)
    ascending = rp.copy()        # (the host check of an upload refuses the others)
    rp[200:3000:301] -= 2 * width + 1  # rows before these are empty, these overlap older entries
    assert _check(gpu, oracle, rp, col, val, ascending)


@pytest.mark.parametrize("N", [70, 137, 4000, 30_000])
@pytest.mark.parametrize("kind", ["far", "alternating", "random", "long_middle", "empty_middle"])
def test_many_diagonals_and_middle_rows(gpu, oracle, N, kind):
    """More diagonals than the list holds, with the middle rows (which are marked
    first and say whether rows share their diagonals) like the others, alternating,
    unlike any other, longer than is looked at, or empty."""
    rng = np.random.default_rng(N)
    step = max(1, N // 80)
    offsets = np.arange(0, min(100, N) * step, step)[:100] if kind != "random" else np.arange(0)
    if kind == "random":
        rows = np.repeat(np.arange(N), 8)
        col = rng.integers(0, N, rows.size)
    else:
        rows = np.repeat(np.arange(N), offsets.size)
        col = (rows + np.tile(offsets, N)) % N
        if kind == "alternating":  # three kinds of rows in turn
            keep = np.tile(np.arange(offsets.size) % 3, N) == rows % 3
            rows, col = rows[keep], col[keep]
    mid = (rows >= N // 2) & (rows < N // 2 + 8)
    if kind in ("long_middle", "empty_middle"):
        rows, col = rows[~mid], col[~mid]
    if kind == "long_middle":
        extra = np.repeat(np.arange(N // 2, min(N, N // 2 + 8)), min(N, 2000))
        rows, col = np.concatenate([rows, extra]), np.concatenate([col, rng.integers(0, N, extra.size)])
    p = np.lexsort((col, rows))
    rows, col = rows[p], col[p]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=N))]).astype(np.int32)
    A = gpu.csr_from_host(rp, col.astype(np.int32), rng.standard_normal(col.size).astype(np.float32))
    for _ in range(3):
        assert gpu.num_diags(A) == [np.unique(col - rows).size, N]

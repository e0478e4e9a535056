"""The analysis's two level kernels against the oracle, bit for bit: the cluster
with the last rows' levels in shared memory (rows that read rows a little
before them) and the tickets over the whole GPU (chains inside a warp, far
dependencies), at the edges of the rule that picks one, of the ring, of a
register group of entries and of a chunk of rows."""
import numpy as np
import pytest

from sciwasm.sparse_b200 import synth

pytestmark = pytest.mark.gpu


def _blocks(N, length):
    """Blocks of `length` rows, each row reading the one before it."""
    i = np.arange(N)
    has = (i % length) != 0
    rp = np.concatenate([[0], np.cumsum(1 + has)]).astype(np.int32)
    col = np.empty(rp[-1], np.int32)
    col[rp[1:] - 1] = i
    col[rp[:-1][has]] = i[has] - 1
    return rp, col, np.ones(col.size)


def _random(N, k, band, seed):
    """Rows of k entries (repeats kept) in the band below and the diagonal."""
    rng = np.random.default_rng(seed)
    i = np.arange(N)
    low = np.maximum(0, i - band)
    c = low[:, None] + (rng.random((N, k)) * (i - low)[:, None]).astype(np.int64)
    col = np.concatenate([np.sort(c, axis=1), i[:, None]], axis=1)
    col[0] = 0
    rp = np.arange(0, N * (k + 1) + 1, k + 1, dtype=np.int32)
    keep = np.ones(col.size, bool)
    keep[:k] = False  # row 0: its diagonal alone
    return (np.concatenate([[0], rp[1:] - k]).astype(np.int32), col.ravel()[keep].astype(np.int32),
            np.ones(N * (k + 1) - k))


def _general(N, seed):
    """Columns on both sides of the diagonal, empty rows, unordered: only
    columns below the row count, and not the last entry."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 12, N)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    row = np.repeat(np.arange(N), lens)
    col = np.clip(row + rng.integers(-700, 300, row.size), 0, N - 1).astype(np.int32)
    return rp, col, rng.uniform(-1, 1, col.size)


CASES = {
    "cluster": lambda: _random(70_001, 7, 900, 1),
    "cluster_smallest": lambda: _random(8192, 7, 1500, 2),
    "below_cluster": lambda: _random(8191, 7, 1500, 2),
    "cluster_long_rows": lambda: _random(30_003, 19, 4000, 3),
    "ring_edge": lambda: _random(60_000, 30, 33_000, 4),
    "near_long_rows": lambda: _random(20_011, 21, 40, 5),
    "far": lambda: _random(90_000, 2, 80_000, 6),
    "laplacian": lambda: synth.laplacian_3d_lower(33),
    "pairs": lambda: _blocks(50_001, 2),
    "warps": lambda: _blocks(50_001, 32),
    "chain": lambda: _blocks(9_000, 9_000),
    "general": lambda: _general(40_000, 7),
}


@pytest.mark.parametrize("name", CASES)
def test_levels_bitexact(gpu, oracle, name):
    rp, col, val = CASES[name]()
    want = oracle.level_sets(rp, col, val)
    for _ in range(2):
        A = gpu.CSR_create_level_sets(gpu.csr_from_host(rp, col, val))
        assert A.nlevels == want["nlevels"]
        assert np.array_equal(A.level_per_row.to_host(), want["level"])
        assert np.array_equal(A.level_index.to_host(), want["level_ptr"])
        assert np.array_equal(A.permutation_index.to_host(), want["permutation"])
        assert np.array_equal(A.order_index.to_host(), want["order"])

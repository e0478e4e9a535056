"""eliminate_zeros of COO and CSR at the edges of the compaction's words (32
entries) and blocks (2048 entries), with rows that are empty, lose every entry
or end on an edge: arrays bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(nnz, kept, dt):
    rng = np.random.default_rng(nnz)
    N = max(nnz // 3, 40)
    cuts = np.sort(rng.integers(0, nnz + 1, N - 1))
    cuts[:3] = 0                                       # leading empty rows
    cuts[-3:] = nnz                                    # trailing ones
    cuts[N // 2:N // 2 + 3] = (nnz // 64) * 32         # rows that begin on a word
    rp = np.concatenate([[0], np.sort(cuts), [nnz]]).astype(np.int32)
    col = rng.integers(0, N, nnz).astype(np.int32)
    val = rng.standard_normal(nnz).astype(dt)
    drop = {"all": 0, "none": nnz, "some": nnz // 2}[kept]
    at = rng.permutation(nnz)[:drop]
    val[at] = np.array([0.0, -0.0, np.nan], dt)[np.arange(drop) % 3]
    if kept == "some":
        val[rng.permutation(nnz)[:3]] = np.array([np.inf, -np.inf, np.finfo(dt).smallest_subnormal])
    return rp, col, val


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("kept", ["some", "all", "none"])
@pytest.mark.parametrize("nnz", [3, 31, 32, 33, 2047, 2048, 2049, 6 * 2048 - 31, 300_001])
def test_compaction_edges(gpu, oracle, nnz, kept, dt):
    rp, col, val = _matrix(nnz, kept, dt)
    N = rp.size - 1
    Z = gpu.eliminate_zeros(gpu.csr_from_host(rp, col, val))
    row = np.repeat(np.arange(N, dtype=np.int32), np.diff(rp))
    ZC = gpu.eliminate_zeros(gpu.coo_from_host(row, col, val, N))
    for got, want in ((Z, oracle.copy_nonzeros_csr(rp, col, val)),
                      (ZC, oracle.copy_nonzeros_coo(row, col, val))):
        assert got.nnz == want[1].size
        assert np.array_equal(got.row_array(), want[0])
        assert np.array_equal(got.col_array(), want[1])
        assert got.val_array().tobytes() == want[2].tobytes()

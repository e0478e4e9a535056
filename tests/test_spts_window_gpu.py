"""Triangular solves on one block with the last rows' values in shared memory
(the window layout of a plan): bit-identical to the oracle's row kernel at the
edges of groups, row lengths and the window, alone and in a batch together
with factors that have no such layout; the reordered CSR comes back out of the
layout bit for bit."""
import numpy as np
import pytest

from sciwasm.sparse_b200 import synth

pytestmark = pytest.mark.gpu


def _ub(a):
    return np.ascontiguousarray(a).view(np.uint8)


def _levels(widths, k, back, dt, seed=5):
    """widths[l] rows at level l; a row reads one row of the level before and
    up to k - 1 more (some rows fewer) of the `back` levels before."""
    rng = np.random.default_rng(seed)
    start = np.concatenate([[0], np.cumsum(widths)])
    rp, col, val = [0], [], []
    for l, w in enumerate(widths):
        for i in range(start[l], start[l + 1]):
            deps = []
            if l and k:
                deps = [rng.integers(start[l - 1], start[l])]
                lo = start[max(0, l - back)]
                deps += list(rng.integers(lo, start[l], rng.integers(k - 1, k + 1) if i % 5 == 0
                                          else k - 1)[:k - 1])
                deps[-1] = lo  # the farthest row in reach
                if len(deps) > 1:
                    deps[0] = rng.integers(start[l - 1], start[l])
                if i % 7 == 3 and len(deps) > 2:
                    deps = deps[:2]
                deps = sorted(set(int(d) for d in deps))
            col += deps + [i]
            val += list(rng.uniform(-0.3, 0.3, len(deps))) + [rng.uniform(2, 4)]
            rp.append(len(col))
    return np.array(rp, np.int32), np.array(col, np.int32), np.array(val, dt)


def _cases(dt):
    slots = (225 * 1024 // np.dtype(dt).itemsize - 1) // 32 * 32  # the widest window
    out = {
        "one_row_levels": _levels([1] * 300, 1, 1, dt),
        "group_edges": _levels([31, 32, 33, 64, 1, 65, 100, 2] * 6, 3, 2, dt),
        "many_groups": _levels([700, 900, 640, 33] * 4, 3, 1, dt),
        "diagonal": _levels([500], 0, 1, dt),
        "at_limit": _levels([32] * (slots // 32 + 40), 2, slots // 32 - 1, dt),
        "past_limit": _levels([32] * (slots // 32 + 40), 2, slots // 32, dt),
    }
    for k in (1, 3, 4, 7, 8, 15, 16):
        out[f"k{k}"] = _levels([40, 70, 33] * 20, k, 3, dt, seed=k)
    out["random"] = synth.random_lower(30_000, seed=4, band=900, dtype=dt)
    return out


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_window_solves_bitexact(gpu, oracle, dt):
    jobs, wants = [], []
    for name, (rp, col, val) in _cases(dt).items():
        N = rp.size - 1
        b = synth.uniform_vec(N, 3, dtype=dt)
        b[:: 11] = -0.0
        want = oracle.spts_csr(rp, col, val, b)
        A = gpu.csr_from_host(rp, col, val)
        bv = gpu.vec_from_host(b)
        ls = oracle.level_sets(rp, col, val)
        R = gpu.CSR_create_level_sets_with_reorder(A)
        assert np.array_equal(R.permutation_index.to_host(), ls["permutation"]), name
        assert np.array_equal(R.row_array(), ls["row_ptr"]), name
        assert np.array_equal(R.col_array(), ls["col"]), name
        assert np.array_equal(_ub(R.val_array()), _ub(ls["val"])), name
        for algo in ("level", "hybrid"):
            yv = gpu.create_vec(N, 0, dt)
            gpu.spts(A, bv, yv, algo=algo)
            assert np.array_equal(_ub(yv.array()), _ub(want)), (name, algo)
        # in place: b and y the same vector
        xv = gpu.vec_from_host(b)
        gpu.spts(A, xv, xv, algo="hybrid")
        assert np.array_equal(_ub(xv.array()), _ub(want)), name
        jobs.append((A._plan, bv.vec_index, gpu.create_vec(N, 0, dt).vec_index))
        wants.append((name, want))
    for own_work in (False, True):
        # (the second batch holds more solves than the GPU has SMs)
        e = gpu.SptsBatch(dt, capacity=20 * len(jobs))
        run = jobs
        if own_work:  # every plan twenty times in one batch
            run = [(p, b, gpu.DeviceArray(b.n, dt), gpu.DeviceArray(b.n, dt))
                   for p, b, _ in jobs * 20]
        for _ in range(2):  # the second run replays the graph
            e.run(run)
            gpu.synchronize()
        assert gpu.sparse._device_status() == 0
        for (name, want), job in zip(wants * 20, run):
            assert np.array_equal(_ub(job[2].to_host()), _ub(want)), (name, own_work)
        # only window layouts, then only the others, then both again
        for pick in (slice(0, 2), slice(5, 6), slice(0, len(jobs))):
            for job in run[pick]:
                job[2].fill_zero()
            e.run(run[pick])
            gpu.synchronize()
            for (name, want), job in list(zip(wants, run))[pick]:
                assert np.array_equal(_ub(job[2].to_host()), _ub(want)), (name, pick)
        e.close()


@pytest.mark.parametrize("dt,policy", [(np.float32, "native"), (np.float32, "f64"),
                                       (np.float64, "native")])
def test_window_solves_special_values(gpu, oracle, dt, policy):
    """Every lane's value is published before its level closes, and values pass
    as they are: infinities and NaN in b and L, zero diagonals (0/0, x/0) in rows
    that others read beside rows padded to their group's length.  Same results
    run after run; NaNs where the oracle has them, other values bit for bit."""
    rng = np.random.default_rng(11)
    rp, col, val = _levels([33, 70, 31, 64, 5] * 30, 7, 3, dt, seed=8)
    N = rp.size - 1
    b = synth.uniform_vec(N, 6, dtype=dt)
    b[rng.integers(0, N, 6)] = [np.inf, -np.inf, np.nan, -0.0, 0.0, np.inf]
    off = np.setdiff1d(np.arange(val.size), rp[1:] - 1)
    val[rng.choice(off, 4, replace=False)] = [np.inf, -np.inf, np.nan, -0.0]
    val[rp[rng.integers(N // 2, N, 3) + 1] - 1] = [0.0, -0.0, np.inf]
    with np.errstate(all="ignore"):
        if policy == "native":
            want = oracle.spts_csr(rp, col, val, b)
        else:  # sums in FP64, each value rounded to FP32 once
            want = np.empty(N, np.float32)
            for i in range(N):
                s, e = rp[i], rp[i + 1] - 1
                t = np.float64(0)
                for j in range(s, e):
                    t = t + np.float64(val[j]) * np.float64(want[col[j]])
                want[i] = np.float32((np.float64(b[i]) - t) / np.float64(val[e]))
    assert np.isnan(want).any() and np.isinf(want).any() and np.isfinite(want).sum() > N // 10
    A, bv, yv = gpu.csr_from_host(rp, col, val), gpu.vec_from_host(b), gpu.create_vec(N, 0, dt)
    nan = np.isnan(want)
    for _ in range(20):
        gpu.spts(A, bv, yv, algo="hybrid", policy=policy)
        y = yv.array()
        assert np.array_equal(np.isnan(y), nan)
        assert np.array_equal(_ub(y[~nan]), _ub(want[~nan]))

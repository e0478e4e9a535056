"""Workloads that time the library through its public entry points.

One pass of a case is what a user's program calls once its matrices are in
device memory: an SpMV, a batch of SpMVs, the conversions between formats,
the structure operations, the level-set analysis and the triangular solves.
Matrices are the banded, 2-D and 3-D Laplacian, power-law, Poisson-row and
random lower-triangular ones that the tests and the benchmark use, made here
on the GPU from the case's seed.  exact() gives the same results in 64 bits
with plain torch.
"""
import math

import numpy as np
import torch

import sciwasm.sparse_b200 as sb

TORCH = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.bfloat16}
NUMPY = {torch.int32: np.int32, torch.float32: np.float32, torch.float64: np.float64,
         torch.bfloat16: np.uint16}
POWER_CAP, POWER_SHIFT = 2000, 15  # row lengths min(cap, Zipf(2) + shift)
POISSON = 12                       # Poisson(12) entries a row, and the diagonal
PER_ROW, BAND = 7, 5000            # random lower factor: entries a row, bandwidth
HALF = 5                           # banded: diagonals -5..5


def listed():
    return [
        # The README's matrix: one small call, where launch latency counts.
        {"name": "spmv_csr_laplacian_256", "kind": "spmv", "matrix": "laplacian", "n": 65536,
         "format": "csr", "dtype": "f32"},
        # A graph-like matrix: skewed rows, random columns, double precision.
        {"name": "spmv_csr_powerlaw_2m", "kind": "spmv", "matrix": "powerlaw", "n": 2000000,
         "format": "csr", "dtype": "f64"},
        # The same kind as it is read from a file, in COO; an odd size.
        {"name": "spmv_coo_powerlaw_777777", "kind": "spmv", "matrix": "powerlaw", "n": 777777,
         "format": "coo", "dtype": "f32"},
        # A large stencil in DIA with its values in 16 bits.
        {"name": "spmv_dia_laplacian_4096_bf16", "kind": "spmv", "matrix": "laplacian",
         "n": 16777216, "format": "dia", "dtype": "bf16"},
        # 512 matrices of 1k to 200k rows with 1 to 8 right-hand sides, one launch.
        {"name": "batch_512", "kind": "batch", "items": 512, "dtype": "f32"},
        # Assembly of a banded matrix from entries in random order.
        {"name": "coo_csr_banded_4m", "kind": "coo_csr", "matrix": "banded", "n": 4000000,
         "dtype": "f64", "shuffled": True},
        # The formats a stencil code goes on with.
        {"name": "csr_dia_ell_banded_4m", "kind": "formats", "matrix": "banded", "n": 4000000,
         "dtype": "f64"},
        # Explicit zeros dropped, then the transpose (A^T of an iterative method).
        {"name": "structure_powerlaw_1m", "kind": "structure", "matrix": "powerlaw", "n": 1000001,
         "dtype": "f32"},
        # Analysis of a new triangular factor.
        {"name": "level_sets_random_1m", "kind": "level_sets", "matrix": "random_lower",
         "n": 1000000, "dtype": "f64"},
        # Solves with an analysed factor: the default algorithm on a factor with
        # many narrow levels, and the level/sync-free hybrid on a stencil's.
        {"name": "spts_level_random_1m", "kind": "spts", "matrix": "random_lower", "n": 1000000,
         "dtype": "f64", "algo": "level", "policy": "native"},
        {"name": "spts_hybrid_laplacian3d_64", "kind": "spts", "matrix": "laplacian3d_lower",
         "n": 262144, "dtype": "f32", "algo": "hybrid", "policy": "native"},
        # A server's batch: factors of both kinds and of many sizes in one launch.
        {"name": "spts_batch_24", "kind": "spts_batch", "items": 24, "largest": 1000000,
         "dtype": "f32", "policy": "native"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("spmv", "spmv", "spmv", "batch", "coo_csr", "formats", "structure",
                       "level_sets", "spts", "spts", "spts_batch"))
    c = {"kind": kind}
    dtype = rng.choice(("f32", "f64"))
    if kind == "spmv":
        c["matrix"] = rng.choice(("laplacian", "banded", "powerlaw"))
        c["n"] = {"laplacian": _log(rng, 32, 4096) ** 2, "banded": _log(rng, 1000, 4000000),
                  "powerlaw": _log(rng, 3000, 2000000)}[c["matrix"]]
        c["format"] = rng.choice(("csr", "coo") if c["matrix"] == "powerlaw"
                                 else ("csr", "coo", "dia", "ell"))
        c["dtype"] = rng.choice(("f32", "f64", "bf16") if c["format"] in ("csr", "dia")
                                else ("f32", "f64"))
    elif kind == "batch":
        c["items"] = _log(rng, 8, 480)
        c["dtype"] = rng.choice(("f32", "bf16"))
    elif kind in ("coo_csr", "formats", "structure"):
        c["matrix"] = rng.choice({"coo_csr": ("banded", "powerlaw"),
                                  "formats": ("banded", "laplacian"),
                                  "structure": ("banded", "powerlaw")}[kind])
        c["n"] = (_log(rng, 32, 2000) ** 2 if c["matrix"] == "laplacian" else
                  _log(rng, 3000, 4000000 if c["matrix"] == "banded" else 1900000))
        c["dtype"] = dtype
        if kind == "coo_csr":
            c["shuffled"] = rng.random() < 0.75
    elif kind in ("level_sets", "spts"):
        c["matrix"] = rng.choice(("random_lower", "laplacian3d_lower"))
        c["n"] = (_log(rng, 1000, 1000000) if c["matrix"] == "random_lower" else
                  _log(rng, 10, 100) ** 3)
        c["dtype"] = dtype
        if kind == "spts":
            c["algo"] = rng.choice(("level", "hybrid", "syncfree"))
            c["policy"] = rng.choice(("native", "f64")) if dtype == "f32" else "native"
    else:
        c["items"] = rng.randint(2, 24)
        c["largest"] = _log(rng, 10000, 1000000)
        c["dtype"] = dtype
        c["policy"] = rng.choice(("native", "f64")) if dtype == "f32" else "native"
    return c


# ---------------------------------------------------------------- inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, gen, dtype=torch.float64):
    return torch.rand(n, generator=gen, device="cuda", dtype=dtype) * 2 - 1


def _row_ptr(counts):
    rp = torch.zeros(counts.numel() + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(counts, 0, out=rp[1:])
    return rp


def _from_keys(key, n):
    """CSR structure of the distinct entries row * n + col, in order."""
    key = torch.unique_consecutive(torch.sort(key)[0])
    row = torch.div(key, n, rounding_mode="floor")
    return _row_ptr(torch.bincount(row, minlength=n)), key - row * n, row


def _stencil(case, gen):
    """offsets, data [diagonals, n] and its mask of a banded matrix or a Laplacian."""
    n = case["n"]
    i = torch.arange(n, device="cuda")
    if case["matrix"] == "banded":
        off = list(range(-HALF, HALF + 1))
        mask = torch.stack([(i + o >= 0) & (i + o < n) for o in off])
        data = torch.randn((len(off), n), generator=gen, device="cuda", dtype=torch.float64)
    else:
        m = math.isqrt(n)
        off = [-m, -1, 0, 1, m]
        mask = torch.stack([i >= m, i % m != 0, i >= 0, i % m != m - 1, i < n - m])
        data = torch.full((5, n), -1.0, device="cuda", dtype=torch.float64)
        data[2] = 4.0
    return off, torch.where(mask, data, 0.0), mask


def _matrix(case, gen):
    """(row_ptr i64, col i64, row i64, val f64) of a case's matrix, rows in order."""
    n, kind = case["n"], case["matrix"]
    if kind in ("banded", "laplacian"):
        off, data, mask = _stencil(case, gen)
        mask = mask.T
        cols = torch.arange(n, device="cuda")[:, None] + torch.tensor(off, device="cuda")
        rp = _row_ptr(mask.sum(1))
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
        return rp, cols[mask], row, data.T[mask]
    if kind == "powerlaw":
        # the row lengths belong to the case, so that every seed gives as many entries
        lens = np.minimum(np.minimum(np.random.default_rng(n).zipf(2.0, n) + POWER_SHIFT, POWER_CAP), n)
        rp = _row_ptr(torch.from_numpy(lens.astype(np.int64)).cuda())
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
        key = row * n + torch.randint(0, n, row.shape, generator=gen, device="cuda")
        while True:  # repeated columns are drawn again
            key = torch.sort(key)[0]
            twice = torch.nonzero(key[1:] == key[:-1]).view(-1)
            if not twice.numel():
                break
            key[twice] = row[twice] * n + torch.randint(0, n, twice.shape, generator=gen, device="cuda")
        return rp, key - row * n, row, _uniform(row.numel(), gen)
    if kind == "laplacian3d_lower":
        m = round(n ** (1 / 3))
        i = torch.arange(n, device="cuda")
        mask = torch.stack([i >= m * m, (i // m) % m != 0, i % m != 0, i >= 0], 1)
        cols = i[:, None] + torch.tensor([-m * m, -m, -1, 0], device="cuda")
        rp, col = _row_ptr(mask.sum(1)), cols[mask]
        row = torch.repeat_interleave(i, rp[1:] - rp[:-1])
        return rp, col, row, torch.where(col == row, 6.0, -1.0).double()
    # random lower factor: distinct columns in the band below, the diagonal last; the
    # structure belongs to the case, so that every seed gives as many levels
    i = torch.arange(n, device="cuda")
    row = torch.repeat_interleave(i, torch.clamp(i, max=PER_ROW))
    lo = torch.clamp(row - BAND, min=0)
    u = torch.rand(row.numel(), generator=_generator(n), device="cuda", dtype=torch.float64)
    col = torch.minimum(lo + (u * (row - lo)).long(), row - 1)
    rp, col, row = _from_keys(torch.cat([row * n + col, i * n + i]), n)
    val = _uniform(col.numel(), gen)
    return rp, col, row, torch.where(col == row, 3.0 + val, 0.5 * val)


def _ell(off, data, mask):
    """Slot k of a row holds its k-th entry; padding is index 0, value 0."""
    i = torch.arange(mask.shape[1], device="cuda").expand(mask.shape)
    at = ((torch.cumsum(mask, 0) - 1)[mask], i[mask])
    ind, dat = torch.zeros_like(mask, dtype=torch.int32), torch.zeros_like(data)
    ind[at] = (i + torch.tensor(off, device="cuda")[:, None])[mask].int()
    dat[at] = data[mask]
    return ind.view(-1), dat.view(-1)


def _array(t):
    return sb.DeviceArray(t.numel(), NUMPY[t.dtype], t.data_ptr())


def _held(obj, *tensors):
    obj.held = tensors  # the object's arrays are these tensors' memory
    return obj


def _csr(rp, col, val, dtype):
    t = (rp.int(), col.int(), val.to(TORCH[dtype]))
    return _held(sb.sparse_CSR_t(*map(_array, t), t[0].numel() - 1, t[1].numel()), *t)


def _coo(row, col, val, n, dtype, rows_sorted):
    t = (row.int(), col.int(), val.to(TORCH[dtype]))
    return _held(sb.sparse_COO_t(*map(_array, t), n, t[0].numel(), rows_sorted=rows_sorted), *t)


def _vec(t):
    return sb.sparse_vec_t(_array(t), t.numel())


def _spmv_inputs(case, seed):
    """The case's matrix object, x and y; and for exact() its entries."""
    gen = _generator(seed)
    n, dt, fmt = case["n"], case["dtype"], case["format"]
    vec = torch.float64 if dt == "f64" else torch.float32
    if fmt in ("dia", "ell"):
        off, data, mask = _stencil(case, gen)
        nnz = int(mask.sum())
        if fmt == "dia":
            t = (torch.tensor(off, device="cuda", dtype=torch.int32), data.to(TORCH[dt]).view(-1))
            A = _held(sb.sparse_DIA_t(*map(_array, t), len(off), n, n, nnz), *t)
            entries = (off, t[1].view(len(off), n), mask)
        else:
            t = _ell(off, data.to(TORCH[dt]), mask)
            A = _held(sb.sparse_ELL_t(*map(_array, t), len(off), n, nnz), *t)
            entries = (off, data.to(TORCH[dt]), mask)
    else:
        rp, col, row, val = _matrix(case, gen)
        A = _csr(rp, col, val, dt) if fmt == "csr" else _coo(row, col, val, n, dt, True)
        entries = (row, col, A.held[2])
    x, y = _uniform(n, gen).to(vec), _uniform(n, gen).to(vec)
    return A, x, y, entries


def _batch_sizes(case):
    """Rows log-uniform in [1000, 200000], right-hand sides 1 to 8 in turn."""
    m = case["items"]
    return [(round(1000 * 200 ** ((k + 0.5) / m)), 1 + 5 * k % 8) for k in range(m)]


def _batch_inputs(case, seed):
    gen = _generator(seed)
    rows = [n for n, _ in _batch_sizes(case)]
    start = np.concatenate([[0], np.cumsum(rows)])
    total = int(start[-1])
    size = torch.repeat_interleave(torch.tensor(rows, device="cuda"), torch.tensor(rows, device="cuda"))
    base = torch.repeat_interleave(torch.tensor(start[:-1], device="cuda"), torch.tensor(rows, device="cuda"))
    counts = torch.poisson(torch.full((total,), float(POISSON), device="cuda"), generator=gen).long()
    row = torch.repeat_interleave(torch.arange(total, device="cuda"), counts)
    u = torch.rand(row.numel(), generator=gen, device="cuda", dtype=torch.float64)
    key = row * total + (u * size[row]).long()
    del u
    own = torch.arange(total, device="cuda")
    key = torch.cat([key, own * total + own - base])
    del row
    rp, col, _ = _from_keys(key, total)
    del key
    val = _uniform(col.numel(), gen, torch.float32)
    jobs = []
    at = rp[torch.tensor(start, device="cuda")].tolist()
    for k, (n, nrhs) in enumerate(_batch_sizes(case)):
        r0, lo, hi = int(start[k]), at[k], at[k + 1]
        A = _csr(rp[r0:r0 + n + 1] - lo, col[lo:hi], val[lo:hi].clone(), case["dtype"])
        jobs.append((A, _uniform(n * nrhs, gen, torch.float32), nrhs))
    return jobs


def _factors(case, seed):
    """Sizes log-uniform up to the largest, 3-D Laplacian and random in turn."""
    gen = _generator(seed)
    m, out = case["items"], []
    for k in range(m):
        n = round(1000 * (case["largest"] / 1000) ** (k / (m - 1)))
        kind = "random_lower" if k % 2 else "laplacian3d_lower"
        n = n if k % 2 else max(10, round(n ** (1 / 3))) ** 3
        rp, col, row, val = _matrix({"matrix": kind, "n": n}, gen)
        out.append((rp, col, row, val.to(TORCH[case["dtype"]]),
                    _uniform(n, gen).to(TORCH[case["dtype"]])))
    return out


def _solve_inputs(case, seed):
    gen = _generator(seed)
    rp, col, row, val = _matrix(case, gen)
    return rp, col, row, val.to(TORCH[case["dtype"]]), _uniform(case["n"], gen).to(TORCH[case["dtype"]])


def _convert_inputs(case, seed):
    """row_ptr and entries; with a tenth of the values zero for "structure"."""
    gen = _generator(seed)
    rp, col, row, val = _matrix(case, gen)
    val = val.to(TORCH[case["dtype"]])
    if case["kind"] == "structure":
        val[torch.randperm(val.numel(), generator=gen, device="cuda")[:val.numel() // 10]] = 0
    if case.get("shuffled"):
        p = torch.randperm(val.numel(), generator=gen, device="cuda")
        row, col, val = row[p], col[p], val[p]
    return rp, col, row, val


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "spmv":
        s["A"], s["x_"], s["out"], _ = _spmv_inputs(case, seed)
        s["x"], s["y"] = _vec(s["x_"]), _vec(s["out"])
    elif kind == "batch":
        s["jobs_"] = _batch_inputs(case, seed)
        # all y in one tensor, each from a multiple of 128 values on
        ends = np.cumsum([-(-x.numel() // 128) * 128 for _, x, _ in s["jobs_"]])
        s["out"] = torch.zeros(int(ends[-1]), device="cuda")
        parts = [(A, _array(x), _array(s["out"][lo:lo + x.numel()]), k)
                 for (A, x, k), lo in zip(s["jobs_"], [0, *ends.tolist()])]
        s["exec"] = sb.BatchExecutor(case["dtype"], capacity=case["items"])
        s["count"] = s["exec"].prepare(parts, overwrite=True)
    elif kind == "coo_csr":
        _, col, row, val = _convert_inputs(case, seed)
        s["A"] = _coo(row, col, val, case["n"], case["dtype"], not case["shuffled"])
    elif kind in ("formats", "structure"):
        rp, col, _, val = _convert_inputs(case, seed)
        s["A"] = _csr(rp, col, val, case["dtype"])
    elif kind in ("level_sets", "spts"):
        rp, col, _, val, b = _solve_inputs(case, seed)
        s["A"] = _csr(rp, col, val, case["dtype"])
        if kind == "spts":
            sb.CSR_create_level_sets(s["A"])
            s["b_"], s["out"] = b, torch.zeros_like(b)
            s["b"], s["y"] = _vec(b), _vec(s["out"])
            s["how"] = (case["algo"], case["policy"])
    else:
        s["jobs"], s["out"] = [], []
        for rp, col, _, val, b in _factors(case, seed):
            A, y = _csr(rp, col, val, case["dtype"]), torch.zeros_like(b)
            s["jobs"].append((_held(sb.SptsPlan(A), b, y), _array(b), _array(y)))
            s["out"].append(y)
        s["exec"] = sb.SptsBatch(NUMPY[TORCH[case["dtype"]]], case["policy"], capacity=case["items"])
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- passes


class _View:
    """A device array's memory for torch, which keeps the array alive."""

    def __init__(self, a):
        self.array = a
        self.__cuda_array_interface__ = {"shape": (a.n,), "typestr": a.dtype.str, "version": 2,
                                         "data": (a.ptr, False)}


def _tensor(a):
    return torch.as_tensor(_View(a), device="cuda")


def _csr_out(A):
    return {"row_ptr": _tensor(A.row_index), "col": _tensor(A.col_index), "val": _tensor(A.val_index)}


def run(s):
    kind = s["kind"]
    if kind == "spmv":
        sb.spmv(s["A"], s["x"], s["y"])
        return s["out"]
    if kind == "batch":
        s["exec"].launch(s["count"])
        return s["out"]
    if kind == "spts":
        sb.spts(s["A"], s["b"], s["y"], *s["how"])
        return s["out"]
    if kind == "spts_batch":
        s["exec"].run(s["jobs"])
        return s["out"]
    if kind == "coo_csr":
        return _csr_out(sb.coo_csr(s["A"]))
    if kind == "formats":
        D, E = sb.csr_dia(s["A"]), sb.csr_ell(s["A"])
        return {"offset": _tensor(D.offset_index), "dia": _tensor(D.data_index),
                "indices": _tensor(E.indices_index), "ell": _tensor(E.data_index)}
    if kind == "structure":
        B = sb.eliminate_zeros(s["A"])
        return {"kept": _csr_out(B), "transposed": _csr_out(sb.transpose(B))}
    R = sb.CSR_create_level_sets_with_reorder(s["A"])
    return dict(_csr_out(R), level=_tensor(R.level_per_row), level_ptr=_tensor(R.level_index),
                perm=_tensor(R.permutation_index), order=_tensor(R.order_index))


# ---------------------------------------------------------------- work and values


def _entries(case):
    """Entries of a case's matrix: counted, or as many as its draw gives on average."""
    n = case["n"]
    if case["matrix"] == "banded":
        return (2 * HALF + 1) * n - HALF * (HALF + 1)
    if case["matrix"] == "laplacian":
        return 5 * n - 4 * math.isqrt(n)
    if case["matrix"] == "laplacian3d_lower":
        return 4 * n - 3 * round(n ** (2 / 3))
    if case["matrix"] == "random_lower":
        return (PER_ROW + 1) * n
    top = POWER_CAP - POWER_SHIFT
    k = np.arange(1, top + 1)
    zipf = 6 / math.pi ** 2
    return int(n * (POWER_SHIFT + zipf * np.sum(1 / k) + top * (1 - zipf * np.sum(1.0 / k ** 2))))


def work(case):
    kind = case["kind"]
    sv = {"f32": 4, "f64": 8, "bf16": 2}[case["dtype"]]
    sx = max(sv, 4)
    if kind == "batch":
        nnz = sum(n * (POISSON + 1) for n, _ in _batch_sizes(case))
        return {"bytes": nnz * (sv + 4) + sum(4 * n + 8 * n * k for n, k in _batch_sizes(case)),
                "flops": sum(2 * n * (POISSON + 1) * k for n, k in _batch_sizes(case))}
    if kind == "spts_batch":
        m, rows, nnz = case["items"], 0, 0
        for k in range(m):
            n = round(1000 * (case["largest"] / 1000) ** (k / (m - 1)))
            rows, nnz = rows + n, nnz + n * (PER_ROW + 1 if k % 2 else 4)
        return {"bytes": nnz * (sv + 4) + rows * (4 + 4 + 2 * sv), "flops": 2 * nnz}
    n, nnz = case["n"], _entries(case)
    csr = nnz * (sv + 4) + 4 * n
    if kind == "spmv":
        matrix = {"csr": csr, "coo": nnz * (sv + 8), "dia": nnz * sv, "ell": nnz * (sv + 4)}
        return {"bytes": matrix[case["format"]] + 3 * n * sx, "flops": 2 * nnz}
    if kind == "coo_csr":
        return {"bytes": nnz * (sv + 8) + csr, "flops": 0}
    if kind == "formats":
        wide = 11 if case["matrix"] == "banded" else 5
        return {"bytes": 2 * csr + wide * n * (2 * sv + 4), "flops": 0}
    if kind == "structure":
        return {"bytes": csr + 3 * (0.9 * nnz * (sv + 4) + 4 * n), "flops": 0}
    if kind == "level_sets":
        return {"bytes": 2 * csr + 4 * 4 * n, "flops": 0}
    return {"bytes": csr + 4 * n + 2 * n * sv, "flops": 2 * nnz}


def _solve(rp, col, row, val, b):
    """Forward substitution as the iteration y = (b - N y) / d over the whole
    factor, whose strictly lower part N is nilpotent."""
    n, val, b = rp.numel() - 1, val.double(), b.double()
    d = val[rp[1:] - 1]
    N = torch.sparse_csr_tensor(rp, col, torch.where(row == col, 0.0, val), size=(n, n))
    y = b / d
    for _ in range(n):
        new = (b - N @ y) / d
        if float((new - y).abs().max()) <= 1e-17 * float(new.abs().max()):
            return new
        y = new
    return y


def _csr_exact(rp, col, val):
    return {"row_ptr": rp.int(), "col": col.int(), "val": val.double()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        _, x, y, entries = _spmv_inputs(case, seed)
        x, y = x.double(), y.double()
        if case["format"] in ("dia", "ell"):
            for o, data, mask in zip(*entries):
                y += torch.where(mask, data.double() * torch.roll(x, -o), 0.0)
            return y
        row, col, val = entries
        return y.index_add_(0, row, val.double() * x[col])
    if kind == "batch":
        out = []
        for A, x, k in _batch_inputs(case, seed):
            rp, col, val = (t.double() if t.dtype != torch.int32 else t.long() for t in A.held)
            row = torch.repeat_interleave(torch.arange(A.N, device="cuda"), rp[1:] - rp[:-1])
            r = torch.zeros((A.N, k), device="cuda", dtype=torch.float64)
            r.index_add_(0, row, val[:, None] * x.double().view(A.N, k)[col])
            out += [r.view(-1), torch.zeros(-r.numel() % 128, device="cuda", dtype=torch.float64)]
        return torch.cat(out)
    if kind == "spts":
        return _solve(*_solve_inputs(case, seed))
    if kind == "spts_batch":
        return [_solve(*f) for f in _factors(case, seed)]
    if kind == "level_sets":
        return None  # indices and copies: nothing is rounded
    rp, col, row, val = _convert_inputs(case, seed)
    n = case["n"]
    if kind == "coo_csr":
        key, p = torch.sort(row * n + col, stable=True)
        return _csr_exact(rp, col[p], val[p])
    if kind == "structure":
        keep = val != 0
        row, col, val = row[keep], col[keep], val[keep]
        p = torch.sort(col, stable=True)[1]
        return {"kept": _csr_exact(_row_ptr(torch.bincount(row, minlength=n)), col, val),
                "transposed": _csr_exact(_row_ptr(torch.bincount(col, minlength=n)), row[p], val[p])}
    off, data, mask = _stencil(case, _generator(seed))
    data = data.to(TORCH[case["dtype"]])
    ind, ell = _ell(off, data, mask)
    return {"offset": torch.tensor(off, device="cuda", dtype=torch.int32),
            "dia": data.double().view(-1), "indices": ind, "ell": ell.double()}

"""Device memory that is kept after sb_free: reuse waits for work in flight on
other streams, blocks are handed out once, double frees are refused, the bound
holds, a failing allocation gives the kept blocks back, and threads may allocate
and free at the same time."""
import ctypes
import threading

import numpy as np
import pytest

from sciwasm.sparse_b200 import _lib

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _alloc(n):
    p = ctypes.c_void_p()
    _lib.call("sb_malloc", ctypes.byref(p), n)
    return p.value


def _info():
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    _lib.call("sb_mem_info", ctypes.byref(free), ctypes.byref(total))
    return free.value, total.value


def test_reuse_waits_for_the_old_use(gpu):
    """A long chain of copies out of a block on one stream; the block is freed
    and allocations of its size follow meanwhile until one gets it, which is
    overwritten on another stream."""
    n = 256 * MIB
    streams = []
    for _ in range(2):
        s = ctypes.c_void_p()
        _lib.call("sb_stream_create", ctypes.byref(s))
        streams.append(s.value)
    src, dst = _alloc(n), _alloc(n)
    others = [_alloc(n) for _ in range(16)]
    _lib.call("sb_stream_synchronize", streams[0])
    _lib.call("sb_memset", src, 0x5A, n, streams[0])
    for _ in range(40):
        _lib.call("sb_memcpy_dtod", dst, src, n, streams[0])
    for p in [src] + others:
        _lib.call("sb_free", p)
    got = []
    while src not in got and len(got) < 64:
        got.append(_alloc(n))
    _lib.call("sb_memset", got[-1], 0, n, streams[1])
    _lib.call("sb_stream_synchronize", streams[0])
    _lib.call("sb_stream_synchronize", streams[1])
    out = np.empty(n, np.uint8)
    _lib.call("sb_memcpy_dtoh", out.ctypes.data, dst, n, None)
    _lib.call("sb_stream_synchronize", None)
    assert np.all(out == 0x5A)
    for p in got + [dst]:
        _lib.call("sb_free", p)
    for s in streams:
        _lib.call("sb_stream_destroy", s)


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
def test_allocation_beside_a_capture(gpu, mode):
    """Blocks are freed and allocated, reused ones too, by this thread while
    another thread captures a stream (thread_local) or this one does (relaxed):
    the capture stays valid."""
    torch = pytest.importorskip("torch")
    n, x = 64 * MIB, torch.zeros(1000, device="cuda")
    g, begun, done = torch.cuda.CUDAGraph(), threading.Event(), threading.Event()
    seen = []

    def churn():
        for _ in range(60):
            seen.append(_alloc(n))
            _lib.call("sb_free", seen[-1])

    def capture(inside):
        with torch.cuda.graph(g, capture_error_mode=mode):
            x.add_(1)
            begun.set()
            inside()
            x.add_(1)

    if mode == "relaxed":
        capture(churn)
    else:
        t = threading.Thread(target=capture, args=(lambda: done.wait(60),))
        t.start()
        begun.wait(60)
        churn()
        done.set()
        t.join()
    g.replay()
    torch.cuda.synchronize()
    assert len(set(seen)) < len(seen) and torch.all(x == 2)


def test_double_free_and_distinct_blocks(gpu):
    lib = _lib.load()
    ps = [_alloc(3 * MIB) for _ in range(4)]
    assert len(set(ps)) == 4
    for p in ps:
        assert lib.sb_free(p) == 0
    assert lib.sb_free(ps[0]) < 0
    qs = [_alloc(3 * MIB) for _ in range(4)]
    assert len(set(qs)) == 4
    for q in qs:
        assert lib.sb_free(q) == 0


def test_bound_and_giving_back(gpu):
    free0, total = _info()
    ps = [_alloc(512 * MIB) for _ in range(8)]
    for p in ps:
        _lib.call("sb_free", p)
    free1, _ = _info()
    assert free1 >= free0 - 64 * MIB  # kept blocks count as free
    big = free1 - 1024 * MIB          # does not fit beside 2 GiB of kept blocks
    p = _alloc(big)
    _lib.call("sb_free", p)
    lib = _lib.load()
    q = ctypes.c_void_p()
    assert lib.sb_malloc(ctypes.byref(q), total * 2) == _lib.SB_ENOMEM and not q.value
    assert lib.sb_malloc(ctypes.byref(q), MIB) == 0
    _lib.call("sb_free", q.value)


def test_threads(gpu):
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        for _ in range(40):
            a = gpu.DeviceArray.from_host(np.full(int(rng.integers(1, 200_000)), seed, np.int32))
            b = gpu.DeviceArray.from_host(np.full(1000, -seed, np.int32))
            if not (np.all(a.to_host() == seed) and np.all(b.to_host() == -seed)):
                bad.append(seed)
            a.free()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(1, 7)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_refused_allocation_is_reported_once(gpu):
    """The launch check of the next call must not see the old error."""
    _, total = _info()
    q = ctypes.c_void_p()
    assert _lib.load().sb_malloc(ctypes.byref(q), total * 2) == _lib.SB_ENOMEM
    A = gpu.csr_from_host(np.array([0, 1, 2]), np.array([0, 1]), np.array([0.0, 3.0]))
    assert gpu.eliminate_zeros(A).nnz == 1


def test_trim_and_bound_as_the_driver_sees_them(gpu):
    """sb_mem_info adds kept bytes to the free ones; here the driver's own figure
    shows how much is kept: 4 GiB at most, and what mem_trim leaves."""
    torch = pytest.importorskip("torch")
    raw = lambda: torch.cuda.mem_get_info()[0]
    gpu.mem_trim()
    free0 = raw()
    ps = [_alloc(512 * MIB) for _ in range(10)]
    assert free0 - raw() >= 10 * 512 * MIB
    for p in ps:
        _lib.call("sb_free", p)
    slack = 64 * MIB
    assert abs(free0 - raw() - 4096 * MIB) <= slack
    gpu.mem_trim(1024 * MIB)
    assert abs(free0 - raw() - 1024 * MIB) <= slack
    assert abs(_info()[0] - raw() - 1024 * MIB) <= slack
    gpu.mem_trim()
    assert abs(free0 - raw()) <= slack and abs(_info()[0] - raw()) <= slack


def test_block_in_use_is_handed_out_after_a_wait(gpu):
    """The kept block that an allocation gets is the one freed while copies out
    of it were queued, and by then they are over: little enough is freed that no
    block goes back to the driver, whose free would wait as well."""
    torch = pytest.importorskip("torch")
    n = 64 * MIB
    gpu.mem_trim()
    streams = []
    for _ in range(2):
        s = ctypes.c_void_p()
        _lib.call("sb_stream_create", ctypes.byref(s))
        streams.append(s.value)
    chain = torch.cuda.ExternalStream(streams[0])
    src, dst = _alloc(n), _alloc(n)
    others = [_alloc(n) for _ in range(16)]
    _lib.call("sb_memset", src, 0x5A, n, streams[0])
    _lib.call("sb_stream_synchronize", streams[0])
    for _ in range(500):
        _lib.call("sb_memcpy_dtod", dst, src, n, streams[0])
    for p in [src] + others:
        _lib.call("sb_free", p)
    assert not chain.query()  # sb_free has not waited
    got = _alloc(n)
    assert got == src and chain.query()
    _lib.call("sb_memset", got, 0, n, streams[1])
    _lib.call("sb_stream_synchronize", streams[1])
    out = np.empty(n, np.uint8)
    _lib.call("sb_memcpy_dtoh", out.ctypes.data, dst, n, None)
    _lib.call("sb_stream_synchronize", None)
    assert np.all(out == 0x5A)
    for p in (got, dst):
        _lib.call("sb_free", p)
    for s in streams:
        _lib.call("sb_stream_destroy", s)

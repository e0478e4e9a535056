"""The rules of the kept device blocks on the host, with a driver that the test
plays: reuse follows a wait, nobody waits for another device, and failed frees
lose no block."""
import os
import subprocess

from sciwasm.sparse_b200 import build

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <future>
#include <set>
#include <thread>
#include "sb_kept_blocks.cuh"
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)

struct Fake {
  using Error = int;
  static inline std::mutex mu;
  static inline std::set<void*> live;
  static inline uintptr_t next = 0x10000;
  static inline size_t used = 0, room = ~size_t(0);
  static inline int mallocs = 0, frees = 0, refuse = 0, waits = 0, beside = 0;
  static inline thread_local bool held_up = false;  // this thread's frees wait for `go`
  static inline std::atomic<int> waiting{0};
  static inline std::promise<void> go;
  static inline std::shared_future<void> gone = go.get_future().share();
  static inline std::unordered_map<void*, size_t> sizes;
  static Error malloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lk(mu);
    if (n > room - used) return 2;
    *p = (void*)(next += 0x1000);
    sizes[*p] = n;
    used += n;
    live.insert(*p);
    ++mallocs;
    return 0;
  }
  static Error free(void* p) {
    if (held_up) {
      ++waiting;
      gone.wait();
    }
    std::lock_guard<std::mutex> lk(mu);
    if (refuse > 0) { --refuse; return 9; }
    if (!live.erase(p)) return 1;
    if (sizes[p] == 16) {  // the waits: cheap only beside another small block
      for (void* q : live) beside += sizes[q] == 16;
      ++waits;
    }
    used -= sizes[p];
    ++frees;
    return 0;
  }
  static Error out_of_memory() { return 2; }
  static void clear() {}
};
using Kept = sb::KeptBlocks<Fake>;
constexpr size_t MIB = 1 << 20;
static void* get(Kept& k, size_t n, int dev = 0) {
  void* p;
  CHECK(k.alloc(&p, n, dev) == 0);
  return p;
}
static void put(Kept& k, void* p) {
  bool twice;
  CHECK(k.free(p, &twice) == 0 && !twice);
}

int main() {
  Kept& k = *new Kept;
  bool twice;
  void* p[17];
  for (void*& q : p) q = get(k, MIB);
  constexpr int few = (int)Kept::kEnoughSame - 1;
  for (int i = 0; i < few; ++i) put(k, p[i]);
  int m = Fake::mallocs, f = Fake::frees;
  void* fresh = get(k, MIB);  // too few of the size: a new block, no wait
  CHECK(Fake::mallocs == m + 1 && Fake::frees == f);
  for (int i = few; i < 17; ++i) put(k, p[i]);
  CHECK(k.free(p[16], &twice) == 0 && twice);
  // enough: the first freed one, after a free by the driver
  std::promise<void*> got;
  std::thread t([&] { Fake::held_up = true; got.set_value(get(k, MIB)); });
  while (!Fake::waiting) std::this_thread::yield();
  // meanwhile: others go on, on this device too; a block freed now was not waited for
  auto rest = std::async(std::launch::async, [&] {
    void* q = get(k, 8 * MIB, 1);
    put(k, q);
    CHECK(k.kept_bytes(1) == 8 * MIB);
    put(k, fresh);
    CHECK(k.kept_bytes(0) == 18 * MIB);
  });
  CHECK(rest.wait_for(std::chrono::seconds(20)) == std::future_status::ready);
  Fake::go.set_value();
  t.join();
  CHECK(got.get_future().get() == p[0]);
  CHECK(Fake::waits == 1 && Fake::beside == 1);
  f = Fake::frees;
  for (int i = 1; i < 17; ++i) CHECK(get(k, MIB) == p[i]);
  CHECK(Fake::frees == f && get(k, MIB) != fresh && k.kept_bytes(0) == MIB);
  // a failed allocation gives everything back and is tried again
  Fake::room = Fake::used + MIB / 2;
  void* big = get(k, MIB + MIB / 4);
  CHECK(k.kept_bytes(0) == 0 && !Fake::live.count(fresh));
  void* none;
  CHECK(k.alloc(&none, 64 * MIB, 0) == 2 && !none);
  Fake::room = ~size_t(0);
  // a free that the driver refuses is reported and loses no block
  put(k, big);
  Fake::refuse = 1;
  CHECK(k.give_back(0, 0, 0) == 9 && k.kept_bytes(0) == MIB + MIB / 4 && Fake::live.count(big));
  CHECK(k.give_back(0, 0, 0) == 0 && k.kept_bytes(0) == 0 && !Fake::live.count(big));
  // the bounds: bytes, and blocks
  void* g[6];
  for (void*& q : g) q = get(k, 1024 * MIB);
  for (void* q : g) put(k, q);
  CHECK(k.kept_bytes(0) == 4096 * MIB && !Fake::live.count(g[1]) && Fake::live.count(g[2]));
  CHECK(k.give_back(0, 0, 0) == 0);
  static void* s[2050];
  for (void*& q : s) q = get(k, 512);
  for (void* q : s) put(k, q);
  CHECK(k.kept_bytes(0) == 2048 * 512);
  // larger than all that is kept: freed at once
  put(k, get(k, 5000 * MIB));
  CHECK(k.kept_bytes(0) == 2048 * 512);
  // sizes that would round up past zero are refused, not granted as nothing
  Fake::room = size_t(1) << 40;
  CHECK(k.alloc(&none, ~size_t(0), 0) == 2 && k.alloc(&none, ~size_t(0) - MIB, 0) == 2);
  CHECK(Kept::round_size(100 * MIB + 1) == 101 * MIB && Kept::round_size(1) == 512);
  // not from here
  CHECK(Fake::malloc(&none, 64) == 0 && k.free(none, &twice) == 0 && !twice);
  std::puts("ok");
}
"""


def test_rules(tmp_path):
    src, exe = tmp_path / "kept.cpp", tmp_path / "kept"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(build.HERE, "csrc"),
                    "-o", exe, src], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.stdout == "ok\n", out.stdout

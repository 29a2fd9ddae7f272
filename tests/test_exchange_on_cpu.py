"""The plain-copy path of the padded exchange kernel, compiled from its own source for the CPU.

The kernel's text (csrc/exchange.cu, up to the bulk-copy path) is built with g++ against stand-ins for the device
primitives, and one block of it after another runs with one host thread per device thread, for one rank of a world
of several.  That shows what one GPU cannot: which scope every counter add has, that all threads of a block meet at
the same barriers, and where the rows for a peer land."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "iris_testing_b200" / "csrc"

PRELUDE = r"""
#include <algorithm>
#include <atomic>
#include <barrier>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>
#include "moe_args.h"
#define __global__
#define __launch_bounds__(...)
#define __shared__ static
#define __syncthreads() sync_at(__LINE__)
using std::min;
struct Dim { int x; };
static thread_local Dim threadIdx, blockIdx;
static Dim blockDim, gridDim;
struct uint4 { uint32_t x, y, z, w; };

// A barrier that notes the source line each thread came from; the first thread runs ahead of the others.
static std::atomic<int> diverged{0};
static std::vector<int> line_of;
struct Compare {
  void operator()() noexcept {
    int seen = 0;
    for (int l : line_of) if (l > 0) { if (seen == 0) seen = l; if (l != seen) diverged = 1; }
  }
};
static std::unique_ptr<std::barrier<Compare>> block_barrier;
static void sync_at(int line) {
  line_of[threadIdx.x] = line;
  block_barrier->arrive_and_wait();
  if (threadIdx.x != 0) std::this_thread::sleep_for(std::chrono::microseconds(300));
}

enum { ST_OVERFLOW = 10, ST_TIMEOUT_BARRIER = 8 };
struct WaitCtx { volatile int* abort_flag; int* status; unsigned long long budget_ns; };
static void report_status(int* status, int code) { if (*status == 0) *status = code; }
static bool wait_flag_geq(const uint32_t* flag, uint32_t target, WaitCtx& w, int code) {
  for (int i = 0; i < 200; ++i) {
    if (__atomic_load_n(flag, __ATOMIC_ACQUIRE) >= target) return true;
    std::this_thread::sleep_for(std::chrono::microseconds(100));
  }
  *w.abort_flag = 1;
  report_status(w.status, code);
  return false;
}
static void chain_wait() {}
static void chain_release() {}
static void mbar_init(uint64_t*, int) {}
static void fence_mbar_init() {}
static void fence_acq_rel_sys() { __atomic_thread_fence(__ATOMIC_SEQ_CST); }
static void fence_acq_rel_gpu() { __atomic_thread_fence(__ATOMIC_SEQ_CST); }
static void st_release_sys(uint32_t* p, uint32_t v) { __atomic_store_n(p, v, __ATOMIC_RELEASE); }
static std::atomic<int> gpu_adds{0}, sys_adds{0};
static void add(uint32_t* p, uint32_t v) { __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
static void red_add_release_sys(uint32_t* p, uint32_t v) { add(p, v); }
static void red_add_relaxed_sys(uint32_t* p, uint32_t v) { ++sys_adds; add(p, v); }
static void red_add_relaxed_gpu(uint32_t* p, uint32_t v) { ++gpu_adds; add(p, v); }
static uint32_t atomicAdd(uint32_t* p, uint32_t v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
static int __ldcg(const int* p) { return *p; }
static uint4 ld_16(const void* p) { uint4 v; memcpy(&v, p, 16); return v; }
static void st_16(void* p, uint4 v) { memcpy(p, &v, 16); }
"""

DRIVER = r"""
template <typename T> static unsigned long long at(std::vector<T>& v) { return reinterpret_cast<unsigned long long>(v.data()); }

int main(int argc, char** argv) {
  const int W = atoi(argv[1]), rank = atoi(argv[2]), EL = atoi(argv[3]), cap = atoi(argv[4]), split = atoi(argv[5]),
            blocks = atoi(argv[6]), mirror = atoi(argv[7]), threads = 64, bm = 4, row_bytes = 48, epoch = 3;
  srand(W * 100 + rank * 10 + EL);
  const int tiles = W * EL * ((cap + bm - 1) / bm);
  std::vector<int> counts(W * EL), dst_off(W), status(1, 0);
  int total = 0;
  for (int d = 0; d < W; ++d) {
    dst_off[d] = total;
    for (int e = 0; e < EL; ++e) { counts[d * EL + e] = rand() % (cap + 1); total += counts[d * EL + e]; }
  }
  // mirror: rows wait in [EL][W][cap] cells and counts are pca[e][src]
  const size_t cells = static_cast<size_t>(EL) * W * cap * row_bytes;
  std::vector<uint8_t> payload(mirror ? cells : static_cast<size_t>(total + 1) * row_bytes);
  for (auto& b : payload) b = static_cast<uint8_t>(rand());
  std::vector<int> pca_local(EL * W);
  for (int e = 0; e < EL; ++e) for (int d = 0; d < W; ++d) pca_local[e * W + d] = counts[d * EL + e];
  std::vector<std::vector<uint8_t>> buf(W, std::vector<uint8_t>(cells, 0));
  std::vector<std::vector<int>> pca(W, std::vector<int>(EL * W, -1));
  std::vector<std::vector<uint32_t>> ready(W, std::vector<uint32_t>(1, 0)), sync(W, std::vector<uint32_t>(std::max(EL, W), 0)),
      entered(W, std::vector<uint32_t>(W, epoch));
  entered[rank][rank] = epoch - 1;           // the kernel itself announces this rank
  sync[rank].assign(sync[rank].size(), mirror ? 0u : 9u);   // left over from the epoch before; re-armed by block 0
  std::vector<uint32_t> parts(2 * tiles, 0);
  PaddedArgs a;
  memset(&a, 0, sizeof(a));
  for (int d = 0; d < W; ++d) {
    a.pca.p[d] = at(pca[d]); a.token_buf.p[d] = at(buf[d]); a.counts_ready.p[d] = at(ready[d]);
    a.token_sync.p[d] = at(sync[d]); a.entered.p[d] = at(entered[d]);
  }
  a.entered_local = entered[rank].data();
  a.epoch = epoch; a.rank = rank; a.world = W; a.e_local = EL; a.cap = cap; a.block_m = bm;
  a.row_bytes = row_bytes; a.mirror = mirror; a.plain = 1; a.split = split;
  a.parts = parts.data(); a.parts_stride = tiles; a.status = status.data(); a.budget_ns = 1000000;
  blockDim.x = threads; gridDim.x = blocks;
  for (int b = 0; b < blocks; ++b) {
    line_of.assign(threads, 0);
    block_barrier.reset(new std::barrier<Compare>(threads));
    std::vector<std::thread> ts;
    for (int t = 0; t < threads; ++t)
      ts.emplace_back([&, t] {
        threadIdx.x = t; blockIdx.x = b;
        padded_bulk_kernel(payload.data(), mirror ? pca_local.data() : counts.data(), mirror ? nullptr : dst_off.data(), a);
        line_of[t] = -1;                     // left the kernel
        block_barrier->arrive_and_drop();
      });
    for (auto& t : ts) t.join();
  }
  int wrong = 0;
  for (int d = 0; d < W; ++d) {
    long long row = mirror ? 0 : dst_off[d];
    unsigned tiles_d = 0;
    for (int e = 0; e < EL; ++e) {
      const int n = counts[d * EL + e];
      const uint8_t* got = buf[d].data() + (mirror ? (static_cast<size_t>(rank) * EL + e) : (static_cast<size_t>(e) * W + rank)) * cap * row_bytes;
      const uint8_t* src = payload.data() + (mirror ? (static_cast<size_t>(e) * W + d) * cap : row) * row_bytes;
      if (memcmp(got, src, static_cast<size_t>(n) * row_bytes) != 0) ++wrong;
      if (!mirror && sync[d][e] != static_cast<unsigned>((n + bm - 1) / bm)) ++wrong;
      if (!mirror && pca[d][e * W + rank] != n) ++wrong;
      tiles_d += (n + bm - 1) / bm;
      row += n;
    }
    if (mirror && sync[d][rank] != tiles_d) ++wrong;
    if (!mirror && ready[d][0] != 1u) ++wrong;
  }
  for (uint32_t p : parts) if (p != 0) ++wrong;
  printf("%d %d %d %d %d\n", wrong, status[0], diverged.load(), gpu_adds.load(), sys_adds.load());
  return 0;
}
"""


@pytest.fixture(scope="module")
def exchange(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src = (CSRC / "exchange.cu").read_text()
    table = re.search(r"struct PeerTable \{.*?\n\};\n", src, re.S).group(0)
    body = src[src.index("constexpr int A2A_WARPS"):src.index("  // ---- tiles: one worker warp per unit")] + "}\n"
    body, n = re.subn(r"  extern __shared__ [^\n]*\n", "", body)
    assert n == 1
    d = tmp_path_factory.mktemp("exchange")
    (d / "x.cpp").write_text(PRELUDE + table + body + DRIVER)
    res = subprocess.run([gxx, "-std=c++20", "-O1", "-w", "-pthread", "-I", str(CSRC), str(d / "x.cpp"), "-o", str(d / "x")],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]

    def run(W, rank, EL, cap, split, blocks, mirror):
        out = subprocess.run([str(d / "x"), *map(str, (W, rank, EL, cap, split, blocks, mirror))], capture_output=True,
                             text=True, timeout=120)
        assert out.returncode == 0, out.stderr
        return dict(zip(("wrong", "status", "diverged", "gpu_adds", "sys_adds"), map(int, out.stdout.split())))
    return run


CASES = [(1, 0, 3, 9, 1, 2, 0), (1, 0, 2, 9, 4, 3, 1), (2, 0, 2, 11, 2, 3, 0), (2, 1, 3, 8, 1, 1, 0), (4, 2, 2, 13, 4, 5, 0),
         (4, 3, 1, 6, 2, 2, 1)]


@pytest.mark.parametrize("W,rank,EL,cap,split,blocks,mirror", CASES)
def test_tile_counters_that_peers_add_to_take_system_scope_adds(exchange, W, rank, EL, cap, split, blocks, mirror):
    """Two adds to one word are atomic towards each other only if each one's scope includes the other thread: a
    counter that other GPUs add to may not be added to at GPU scope here."""
    r = exchange(W, rank, EL, cap, split, blocks, mirror)
    assert r["gpu_adds"] == 0 and r["sys_adds"] > 0, r


def test_no_kernel_adds_to_a_flag_at_gpu_scope():
    """The same for every kernel, by the source: the counters in symmetric memory are added to by several ranks."""
    for f in sorted(CSRC.glob("*.cu*")):
        assert not re.search(r"red\.\w+\.gpu\b|red_add_\w+_gpu\b", f.read_text()), f.name


@pytest.mark.parametrize("W,rank,EL,cap,split,blocks,mirror", CASES + [(8, 5, 2, 9, 2, 2, 0)])
def test_threads_of_a_block_meet_at_the_same_barriers(exchange, W, rank, EL, cap, split, blocks, mirror):
    """One thread waits for a peer on behalf of its block; whether the block waits must be decided alike by threads
    that run ahead and threads that come late.  Rows, counts and flags land where they belong, none twice."""
    r = exchange(W, rank, EL, cap, split, blocks, mirror)
    assert r["diverged"] == 0 and r["wrong"] == 0 and r["status"] == 0, r

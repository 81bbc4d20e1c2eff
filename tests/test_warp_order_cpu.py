"""Order of memory between the lanes of a warp, on the CPU: a kernel's text is compiled for the host, its lanes are threads,
and what a lane stores to shared memory stays its own until the next __syncwarp(), since that is all that the CUDA
programming model promises: shuffles bring lanes together but order no memory."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <pthread.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <thread>
#include <unordered_map>
#include <vector>
typedef uint32_t u32;
typedef uint64_t u64;
using std::min;
#define __global__
#define __launch_bounds__(...)
struct Dim { u32 x; };
thread_local Dim threadIdx, blockIdx;
pthread_barrier_t meet;
struct Word;
thread_local std::unordered_map<Word*, u32> own;   // stores that no __syncwarp has published
struct Word {
  u32 seen;
  operator u32() { const auto it = own.find(this); return it == own.end() ? seen : it->second; }
  u32 operator=(u32 x) { own[this] = x; return x; }
};
Word shared_words[1 << 16];
u32 exchange[32];
void together() { pthread_barrier_wait(&meet); }
void __syncwarp() {
  together();
  for (auto& o : own) o.first->seen = o.second;
  own.clear();
  together();
}
u32 __shfl_sync(u32, u32 v, u32 from) {
  exchange[threadIdx.x & 31] = v;
  together();
  const u32 r = exchange[from & 31];
  together();
  return r;
}
u32 __ldg(const u32* p) { return *p; }
struct Rand4 { u32 x, y, z, w; };
enum { TAG_WALK, SKW_APP_DEEPWALK, SKW_APP_PPR };
const u32 kNoVertex = 0xFFFFFFFFu;
const u32 kWalkCta = 64;
struct WalkArgs {
  const u32* starts;
  u32 *paths, *lengths;
  u64* sum;
  u64 seed, n, walker_base, walker_stride;
  u32 hop_num;
};
Rand4 philox_tagged(u64 seed, int, u64 walker, u32 step, u32) {
  u64 h = (seed + walker * 1000003 + step) * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  h *= 0xBF58476D1CE4E5B9ull;
  return Rand4{(u32)(h >> 32), (u32)h, (u32)(h >> 16), 0};
}
template <int APP, bool AHEAD>
bool walk_step(const WalkArgs&, u32, u64, u32 cur, u32& next, Rand4 r) {
  next = cur * 5 + r.x % 1000;
  return r.y % 64 != 0;
}
void add_edges(u64* sum, u64 mine) { __atomic_fetch_add(sum, mine, __ATOMIC_RELAXED); }
"""

MAIN = r"""
template <int APP>
int check(u32 n, u32 hop, u32 lanes, u32 off) {
  std::vector<u32> room(32 + off + n * hop + 64, 7u), lengths(n, 7u), starts(n);
  u32* const line = reinterpret_cast<u32*>((reinterpret_cast<uintptr_t>(room.data()) + 127) & ~(uintptr_t)127);
  u32* const rows = line + off;
  for (u32 w = 0; w < n; ++w) starts[w] = w * 11;
  u64 sum = 0;
  const WalkArgs a{starts.data(), rows, lengths.data(), &sum, 17, n, 3, 2, hop};
  const u32 warps = (n + lanes - 1) / lanes;
  for (u32 warp = 0; warp < (warps + 1) / 2 * 2; ++warp) {
    std::vector<std::thread> ts;
    for (u32 lane = 0; lane < 32; ++lane)
      ts.emplace_back([&, lane] {
        blockIdx.x = warp / 2;
        threadIdx.x = (warp & 1) * 32 + lane;
        own.clear();
        walk_home_kernel<APP, true>(a, lanes);
      });
    for (auto& t : ts) t.join();
  }
  u64 edges = 0;
  for (u32 w = 0; w < n; ++w) {
    u32 cur = starts[w], len = 0;
    bool live = true;
    for (u32 c = 0; c < hop; ++c) {
      const u32 want = live ? cur : kNoVertex;
      if (rows[(u64)w * hop + c] != want) return printf("n %u hop %u lanes %u off %u: walker %u cell %u\n", n, hop, lanes, off, w, c), 1;
      u32 next;
      if (live && c + 1 < hop && (live = walk_step<APP, true>(a, c, 0, cur, next, philox_tagged(17, TAG_WALK, 3 + 2ull * w, c, 0)))) cur = next, ++len;
    }
    if (lengths[w] != len) return printf("length of walker %u\n", w), 1;
    edges += len;
  }
  for (u32* p = rows + (u64)n * hop; p < room.data() + room.size(); ++p)
    if (*p != 7u) return puts("behind the rows"), 1;
  return sum != edges;
}
int main() {
  pthread_barrier_init(&meet, nullptr, 32);
  int bad = 0;
  for (u32 hop : {1u, 31u, 33u, 70u})
    bad += check<SKW_APP_DEEPWALK>(5, hop, 1, 3) + check<SKW_APP_PPR>(9, hop, 4, 31) + check<SKW_APP_DEEPWALK>(37, hop, 32, 0);
  return bad != 0;
}
"""


def test_rows_written_home_wait_for_the_cells(tmp_path):
    """walk_home_kernel: every lane puts its walker's cells into shared memory, then all lanes write all rows from there."""
    src = open(os.path.join(ROOT, "skywalker_b200", "csrc", "skw_walk.cu")).read()
    kernel = re.search(r"constexpr u32 kLineCells = .*?\n}\n", src, re.S).group(0)
    assert "walk_home_kernel" in kernel
    for was, becomes in (("extern __shared__ u32 rings[];", "Word* const rings = shared_words;"),
                         ("u32* const warp_rings", "Word* const warp_rings"), ("u32* const ring ", "Word* const ring ")):
        assert kernel.count(was) == 1
        kernel = kernel.replace(was, becomes)
    cpp, exe = tmp_path / "home.cpp", tmp_path / "home"
    cpp.write_text(SHIM + kernel + MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", str(cpp), "-o", str(exe)], check=True, timeout=300)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout

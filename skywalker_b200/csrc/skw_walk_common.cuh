// Shared by the walk kernels: launch arguments, the connectivity test of node2vec, the edge counter.
#pragma once
#include "skw_ctx.h"

namespace skw {

constexpr u32 kAlive = 0xFFFFFFFFu;
constexpr u32 kNoVertex = 0xFFFFFFFFu;
constexpr u32 kN2vMaxTrials = 64;

struct WalkArgs {
  const u32* xadj;
  const u32* adjncy;
  const Slot* slots;
  const u32* starts;
  u32* paths;
  u32* lengths;
  unsigned long long* sum;
  u32* err;
  u64 n;
  u64 seed;
  u64 walker_base;
  u64 walker_stride;
  u32 V;
  u32 hop_num;
  u32 unbiased;  // uniform neighbour choice: no table is read
  float tp, inv_p, inv_q, fmax;
};

// bool CheckConnect(src, dst) of the reference (include/gpu_graph.cuh:204-238): whether dst is in the sorted
// list adjncy[lo, hi).  A lane searching alone is a chain of dependent accesses, each of which costs the same
// for 4 or 32 bytes, so a round loads the whole 32-byte sector at the place where dst should be if the ids of
// the list were spread evenly between the values known at its ends.  Ids mostly are (they are names, not
// ranks), and two or three rounds then do what a binary search of 3,700 entries does in twelve; from the fourth
// round on every other one halves the list instead, so that no list takes more than twice the halvings.
struct ListSearch {
  u32 lo, hi;    // dst, if present, lies in adjncy[lo, hi) ...
  u32 vlo, vhi;  // ... whose values lie in [vlo, vhi)
  u32 round;
  __device__ __forceinline__ ListSearch() {}
  __device__ __forceinline__ ListSearch(u32 first, u32 end, u32 V) : lo(first), hi(end), vlo(0), vhi(V), round(0) {}
  // First entry of the sector to load next (lo < hi and vlo <= dst < vhi hold).
  __device__ __forceinline__ u32 sector(u32 dst) const {
    const u32 span = hi - lo;
    const float at = __fdividef((float)(dst - vlo), (float)(vhi - vlo)) * (float)span;
    const u32 step = round >= 3 && (round & 1) ? span >> 1 : (u32)at;
    return (lo + min(step, span - 1)) & ~7u;
  }
  // Takes in entries s .. s + 7; true when the search is over (hit tells its outcome).
  __device__ __forceinline__ bool advance(const u32 (&x)[8], u32 s, u32 dst, bool& hit) {
    hit = false;
    u32 below = 0;
#pragma unroll
    for (u32 k = 0; k < 8; ++k) {
      const bool in = s + k >= lo && s + k < hi;
      hit |= in && x[k] == dst;
      below += in && x[k] < dst ? 1u : 0u;
    }
    const u32 a = max(s, lo), b = hi - s > 8 ? s + 8 : hi;
    if (hit || (below != 0 && below != b - a)) return true;
    ++round;
    if (below == 0) {
      hi = a;
      if (a == s) vhi = x[0];
    } else {
      lo = b;
      if (b == s + 8) vlo = x[7] + 1;
    }
    return lo >= hi || vlo > dst || vhi <= dst;
  }
};
// The sector of eight entries from s on; `wide`: the array starts on a 32-byte boundary, so that a sector with an entry of
// the list in it lies in one page with that entry, also where the array ends inside it.
__device__ __forceinline__ void load_sector(const u32* __restrict__ adjncy, u32 s, u32 lo, u32 hi, bool wide, u32 (&x)[8]) {
  if (wide) {
    asm volatile("ld.global.nc.L1::no_allocate.L2::64B.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
                 : "l"(adjncy + s));
  } else {
#pragma unroll
    for (u32 k = 0; k < 8; ++k) x[k] = __ldg(adjncy + min(max(s + k, lo), hi - 1));
  }
}
__device__ __forceinline__ bool on_sector_boundary(const u32* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }
__device__ __forceinline__ bool connected(const u32* __restrict__ adjncy, u32 lo, u32 hi, u32 dst, u32 V) {
  ListSearch f(lo, hi, V);
  bool hit = false;
  for (bool over = lo >= hi; !over;) {
    u32 x[8];
    const u32 s = f.sector(dst);
    load_sector(adjncy, s, f.lo, f.hi, on_sector_boundary(adjncy), x);
    over = f.advance(x, s, dst, hit);
  }
  return hit;
}

// The same by halving the list: more accesses, a third of the instructions of a round each.
__device__ __forceinline__ bool connected_by_halving(const u32* __restrict__ adjncy, u32 lo, u32 hi, u32 dst) {
  while (lo < hi) {
    const u32 mid = lo + ((hi - lo) >> 1);
    const u32 x = __ldg(adjncy + mid);
    if (x == dst) return true;
    if (x < dst) lo = mid + 1;
    else hi = mid;
  }
  return false;
}

// Whether node2vec keeps a proposal: x = u * max(1/p, 1, 1/q) lies below f, where f is 1/p for the vertex
// the walk came from, 1 for a neighbour of that vertex and 1/q for any other.  The list of that vertex is
// searched (linked()) only when the answer depends on it: below both 1 and 1/q the proposal is kept, at
// or above both it is not (p = 2, q = 0.5: half of the proposals are decided without a search).
template <class Linked>
__device__ __forceinline__ bool n2v_keep(float x, bool back, float inv_p, float inv_q, Linked linked) {
  if (back) return x < inv_p;
  if (x < fminf(1.0f, inv_q)) return true;
  if (!(x < fmaxf(1.0f, inv_q))) return false;
  return linked() ? x < 1.0f : x < inv_q;
}

__device__ __forceinline__ void add_edges(unsigned long long* sum, u64 edges) {
#pragma unroll
  for (int o = 16; o; o >>= 1) edges += __shfl_xor_sync(0xFFFFFFFFu, edges, o);
  if ((threadIdx.x & 31) == 0 && edges) atomicAdd(sum, (unsigned long long)edges);
}

// One warp per walker, every step's slot computed from the weight list (skw_walk_direct.cu).
int launch_walk_online_direct(skw_ctx* ctx, const WalkArgs& a, uint32_t app);

}  // namespace skw

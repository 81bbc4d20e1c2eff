// Offline alias-table construction for all vertices of a range.
//
// Takes over ConstructTable / ConstructAliasTableKernel (src/createTable.cu:48-179 of the
// reference) and the alias_table_constructor_shmem methods it drives (loadFromGraph, construct,
// constructBC, SaveAliasTable; include/alias_table_new.cuh:1077-1132, 1211-1316, 334-464,
// 1105-1115).
//
// Construction rule (one vertex, degree n, weights w_0..w_{n-1}; identical to the sequential
// sweep "smalls in index order are topped up by larges in index order, a large that falls below
// one bucket is topped up by the next large"):
//   masses    B = min(40, 62 - ceil(log2 n)), C = 2^B, q_i = trunc(w_i * 2^(B-1-e)) with
//             e = floor(log2 max w), Q_i = q_0 + .. + q_(i-1), W = Q_n, K = n*C / W (one IEEE
//             double division), g(Q) = n*C if Q == W else min(n*C, trunc((double)Q * K)),
//             M_i = g(Q_i + q_i) - g(Q_i).  g is monotone, so zero weights get zero mass and
//             sum M_i == n*C exactly.
//   classes   small: M_i < C, large: M_i >= C.
//   prefixes  D(i) = sum over smalls at positions <= i of (C - M), X(i) = sum over larges at
//             positions <= i of (M - C)   (both over list positions, zeros elsewhere).
//   small s   alias = first large l at or after the first position with X >= D(s) - (C - M_s),
//             prob  = M_s / C.
//   large l   let S = first position with D(S) > X(l); if none: prob = 1, alias = l; else
//             prob = (X(l) + C - D(S)) / C, alias = next large after l.
// Every quantity is an integer or a single correctly rounded IEEE operation, so the table is a
// pure function of the weight list: no atomics on masses, no dependence on scheduling.
//
// Work distribution: vertices are binned by degree with warp ballots and shared-memory prefix sums (classify_*
// kernels), one work list per class.  Lists of up to 4096 weights are built in double precision by a lane, a group of
// lanes, a warp or a CTA that holds the whole list in registers (skw_alias_f64.cuh), up to 16384 by a CTA alike
// (skw_alias_wide.cuh); longer ones are worked through in tiles (skw_alias_long.cuh) by teams of CTAs, clusters of eight, four
// or two or CTAs alone by the number of lists, and beyond 65536 always by eight.
#include <math_constants.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "skw_alias_f64.cuh"
#include "skw_alias_long.cuh"
#include "skw_alias_math.cuh"
#include "skw_alias_wide.cuh"
#include "skw_ctx.h"

namespace skw {

// Degree classes.  Up to 4096 weights a list is one tile in the registers of NT threads, EPT weights each
// (skw_alias_f64.cuh): one lane with 8 or 16; groups of 2 to 32 lanes and CTAs of 64 to 256 threads with 16.  What a
// thread spends on scans, the division and its way into the merge (some 300 instructions) is shared by its weights,
// so few threads with many weights beat many with few.  Up to 16384 a list is still one tile, of a CTA of 512 or 1024 threads
// (skw_alias_wide.cuh).  Longer ones are worked through in tiles, with the entries in global scratch (skw_alias_long.cuh).
enum { K_1A = 0, K_1B, K_2, K_4, K_8, K_16, K_32, K_C64, K_C128, K_C256, K_C2A, K_C2, K_H, K_G, K_CLASSES };
constexpr u32 kListEpt = 16;
constexpr u32 kGroupMax = 32 * kListEpt;      // 512: the longest list of a group of lanes
constexpr u32 kMidSmemMax = 512 * kWideEpt;   // 8192: two CTAs of 512 threads an SM, 84 KB of lists each
constexpr u32 kHugeSmemMax = 1024 * kWideEpt;  // 16384: one of 1024 threads; longer lists are in global memory
constexpr u32 kAloneMax = skw_ctx::kLongMost;  // longer ones are always built by clusters
static_assert(kHugeSmemMax + 1 == skw_ctx::kLongLeast, "the graph's lists of class K_H are counted");
static_assert(256 * kListEpt == kF64Max, "the classes up to 4096 end where the packed entries end");
static_assert(2 * K_CLASSES <= skw_ctx::kClassWords, "class counters");

__device__ __forceinline__ int degree_class(u32 deg) {
  if (deg <= 8) return K_1A;
  if (deg <= kF64Max) return deg <= kListEpt ? K_1B : K_1B + (32 - __clz((int)((deg - 1) / kListEpt)));
  if (deg <= kMidSmemMax) return K_C2A;
  if (deg <= kHugeSmemMax) return K_C2;
  return deg <= kAloneMax ? K_H : K_G;
}

// The work list of every class: vertices of that class in no particular order, cls[k] of them; cls[K + k] is the
// cursor from which the kernels of the long lists take their next vertex.
struct ClassLists {
  u32* list[K_CLASSES];
};

// One pass over the offsets: a tile of 1024 vertices is binned with ballots, its counts reserve room in the lists with
// one atomic per class and tile, and the vertices are written there.  Each list has room for as many vertices of its
// least degree as there can be edges for (class_room), so nothing has to be counted first: reading the offsets once
// instead of twice took the classification of 16.8 M vertices from 304 to 120 us.
constexpr u32 kClassifyVertices = 4;  // per thread
__global__ void __launch_bounds__(256) classify_kernel(const u32* __restrict__ xadj, u32 v_begin, u32 v_end,
                                                       u32* __restrict__ cls, const ClassLists lists,
                                                       uint8_t* __restrict__ valid) {
  __shared__ u32 s_cnt[K_CLASSES], s_base[K_CLASSES];
  const u32 lane = threadIdx.x & 31;
  constexpr u32 kTile = 256 * kClassifyVertices;
  for (u64 v0 = v_begin + (u64)blockIdx.x * kTile; v0 < v_end; v0 += (u64)gridDim.x * kTile) {
    if (threadIdx.x < K_CLASSES) s_cnt[threadIdx.x] = 0;
    int c[kClassifyVertices];
    u32 rank[kClassifyVertices];
#pragma unroll
    for (u32 j = 0; j < kClassifyVertices; ++j) {
      const u64 v = v0 + j * 256 + threadIdx.x;
      c[j] = -1;
      if (v < v_end) {
        const u32 deg = __ldg(xadj + v + 1) - __ldg(xadj + v);
        if (deg == 0) valid[v] = 0;
        else c[j] = degree_class(deg);
      }
    }
    __syncthreads();
#pragma unroll
    for (u32 j = 0; j < kClassifyVertices; ++j) {
      const u32 same = __match_any_sync(0xFFFFFFFFu, c[j]);
      const int first = __ffs(same) - 1;
      u32 at = 0;
      if (c[j] >= 0 && lane == (u32)first) at = atomicAdd(&s_cnt[c[j]], (u32)__popc(same));
      rank[j] = __shfl_sync(0xFFFFFFFFu, at, first) + __popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (threadIdx.x < K_CLASSES && s_cnt[threadIdx.x]) s_base[threadIdx.x] = atomicAdd(&cls[threadIdx.x], s_cnt[threadIdx.x]);
    __syncthreads();
#pragma unroll
    for (u32 j = 0; j < kClassifyVertices; ++j)
      if (c[j] >= 0) lists.list[c[j]][s_base[c[j]] + rank[j]] = (u32)(v0 + j * 256 + threadIdx.x);
    __syncthreads();
  }
}

// Vertices that class k can have at most, with E edges on V vertices.
static u64 class_room(int k, u64 V, u64 E) {
  static const u32 least[K_CLASSES] = {1, 9, 17, 33, 65, 129, 257, 513, 1025, 2049, kF64Max + 1, kMidSmemMax + 1, kHugeSmemMax + 1,
                                       kAloneMax + 1};
  return std::min<u64>(V, E / least[k]) + 1;
}

// ------------------------------------------------------------------ bounded wait ----------
// (of the self-test; the builders wait for nothing)
__device__ __forceinline__ u32 smem_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(u64* bar, u32 arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Poll (without blocking) for the phase with the given parity, at most `limit` times with a short
// sleep in between: a few milliseconds in total.  Returns false if the copy did not complete.
__device__ __forceinline__ bool mbar_wait(u64* bar, u32 parity, u32 limit) {
  for (u32 i = 0; i < limit; ++i) {
    u32 done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    __nanosleep(32);
  }
  return false;
}

// ------------------------------------------------------------------ lists of up to 4096 ----
// The vertices of one class that a group, warp or CTA works through: items first, first + stride ... of the class's
// work list.  A vertex is reached by a chain of three dependent accesses (work list, offsets, weights), which is
// longer than the building of a short list: so the list is read three items ahead, the offsets two, and the
// weights of the next item are on their way to L2 while this one is built.
struct ClassItems {
  const u32* list;  // at the current item
  const u32* xadj;
  u32 left, stride;        // items from the current one on
  u32 v, off, end;         // the current item
  u32 v1, off1, end1, v2;  // the next one; the vertex after it
  struct After {
    u32 off2, end2, v3;
  };
  __device__ __forceinline__ u32 vertex(u32 steps) const { return left > steps * stride ? __ldg(list + steps * stride) : 0u; }
  __device__ __forceinline__ ClassItems(const u32* all, u32 count, const u32* x, u32 first, u32 step)
      : list(all + first), xadj(x), left(count - min(count, first)), stride(step) {
    v = vertex(0);
    v1 = vertex(1);
    v2 = vertex(2);
    off = __ldg(xadj + v);
    end = __ldg(xadj + v + 1);
    off1 = __ldg(xadj + v1);
    end1 = __ldg(xadj + v1 + 1);
  }
  __device__ __forceinline__ bool more() const { return left != 0; }
  // Called before the current item is built; advance() takes what it returns.  Thread t brings in the weights of
  // the next item from per_thread * t on.
  __device__ __forceinline__ After look_ahead(const float* wgt, u32 t, u32 per_thread) const {
    if (left > stride && t * per_thread < end1 - off1)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(wgt + off1 + t * per_thread));
    return After{__ldg(xadj + v2), __ldg(xadj + v2 + 1), vertex(3)};
  }
  __device__ __forceinline__ void advance(const After& a) {
    left -= min(left, stride);
    list += stride;
    v = v1;
    off = off1;
    end = end1;
    v1 = v2;
    off1 = a.off2;
    end1 = a.end2;
    v2 = a.v3;
  }
};

// Shared memory of one vertex, and of a warp that has 32 / G of them side by side.
template <int G, int EPT>
struct GroupShared {
  // an odd number of words a group; the slots also hold the staged weights (G >= 8: n + n / EPT words of 4 bytes)
  static constexpr u32 kWords = (G * EPT + 1) | 1;
  uint2 lists[32 / G][kWords], slots[32 / G][kWords];
};
template <int NT>
struct ListShared {
  uint2 list[NT * kListEpt + 2], slots[NT * kListEpt];
  typename CtaCoop<NT>::Words words;
};
// bytes a warp has, whatever class it is at
constexpr size_t kWarpBytes =
    (std::max({sizeof(GroupShared<32, 16>), sizeof(GroupShared<16, 16>), sizeof(GroupShared<8, 16>),
               sizeof(GroupShared<4, 16>), sizeof(GroupShared<2, 16>), sizeof(GroupShared<1, 16>),
               (sizeof(ListShared<64>) + 1) / 2, (sizeof(ListShared<128>) + 3) / 4, (sizeof(ListShared<256>) + 7) / 8}) + 15) / 16 * 16;
constexpr u32 kListWarps = 8, kListCtas = 3;  // warps a CTA, CTAs an SM: what registers and shared memory allow

struct ListBuild {
  const u32* xadj;
  const float* wgt;
  Slot* slots;
  uint8_t* valid;
  u32* err;
};

// The lists of one class, NT threads each with up to EPT weights a thread.  `turn` is where in the row of all warps the
// class starts: classes are dealt out one behind the other, so that the few lists of a small graph go to different warps.
// Moved on to the end of this class.
template <int NT, int EPT>
__device__ __forceinline__ void build_class(const ListBuild& b, unsigned char* smem, const u32* list, u32 count, u32& turn) {
  const u32 warps = gridDim.x * kListWarps;
  const u32 workers = NT >= 32 ? warps / (NT / 32) : warps * (32 / NT);
  const u32 me = (blockIdx.x * (kListWarps * 32) + threadIdx.x) / NT;
  const u32 start = NT >= 32 ? turn / (NT / 32) : turn * (32 / NT);
  const u32 first = me >= start ? me - start : me + workers - start;
  turn = (u32)((turn + ((u64)count * NT + 31) / 32) % warps);
  auto build = [&](const auto& co, uint2* A, uint2* out) {
    for (ClassItems c(list, count, b.xadj, first, workers); c.more();) {
      const ClassItems::After after = c.look_ahead(b.wgt, co.t, NT >= 8 ? 32 : EPT);
      const u32 n = c.end - c.off;
      if (n > NT * EPT || n == 0) {  // classification and kernel disagree: record and skip
        if (co.t == 0) dev_fail(b.err, DEV_ERR_INTERNAL, c.v, n, NT);
      } else {
        build_list_f64<std::decay_t<decltype(co)>, EPT>(co, c.v, c.off, n, b.wgt + c.off, b.slots, b.valid, A, out, b.err);
      }
      co.sync();  // the words are reused by the next vertex
      c.advance(after);
    }
  };
  if constexpr (NT <= 32) {
    GroupShared<NT, EPT>* sh = reinterpret_cast<GroupShared<NT, EPT>*>(smem + (threadIdx.x >> 5) * kWarpBytes);
    const u32 in_warp = (threadIdx.x & 31) / NT;
    if (first < count) build(GroupCoop<NT>(), sh->lists[in_warp], sh->slots[in_warp]);
    __syncwarp();
  } else {
    const u32 part = threadIdx.x / NT;
    ListShared<NT>* sh = reinterpret_cast<ListShared<NT>*>(smem + part * (NT / 32) * kWarpBytes);
    if (first < count) build(CtaCoop<NT>(&sh->words, part), sh->list, sh->slots);
  }
}

// Lists of up to 4096 weights: a CTA's warps work together or in parts on those of more than 512 (LONGER), alone or with
// several lists side by side on the others.  Nothing orders the classes.  As launches of their own they cost a small graph
// 9 us each, with every warp going through all of them in turn 53 us (1 M edges); dealt out one behind the other 24 us.
// All in one kernel cost more registers than there are: 7 % slower on large graphs.
template <bool LONGER>
__global__ void __launch_bounds__(kListWarps * 32, kListCtas)
    build_lists_kernel(const ClassLists lists, const u32* __restrict__ cls, const __grid_constant__ ListBuild b) {
  extern __shared__ __align__(16) unsigned char smem[];
  u32 turn = 0;
  if constexpr (LONGER) {
    build_class<256, 16>(b, smem, lists.list[K_C256], cls[K_C256], turn);
    build_class<128, 16>(b, smem, lists.list[K_C128], cls[K_C128], turn);
    build_class<64, 16>(b, smem, lists.list[K_C64], cls[K_C64], turn);
  } else {
    build_class<32, 16>(b, smem, lists.list[K_32], cls[K_32], turn);
    build_class<16, 16>(b, smem, lists.list[K_16], cls[K_16], turn);
    build_class<8, 16>(b, smem, lists.list[K_8], cls[K_8], turn);
    build_class<4, 16>(b, smem, lists.list[K_4], cls[K_4], turn);
    build_class<2, 16>(b, smem, lists.list[K_2], cls[K_2], turn);
    build_class<1, 16>(b, smem, lists.list[K_1B], cls[K_1B], turn);
    build_class<1, 8>(b, smem, lists.list[K_1A], cls[K_1A], turn);
  }
}

// 4097 to 16384 weights: a CTA a list.
template <u32 NT>
__global__ void __launch_bounds__(NT, 1024 / NT) build_wide_kernel(const u32* __restrict__ list, u32* __restrict__ cls, int k,
                                                                   const __grid_constant__ ListBuild b) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ u32 s_next;
  WideItems items{list, b.xadj, b.wgt, cls + K_CLASSES + k, cls[k], &s_next};
  if (items.count == 0) return;
  items.ask();
  items.tell();
  __syncthreads();
  items.vertex();
  if (!items.more) return;
  items.offsets();
  items.advance();
  for (;;) {
    items.ask();
    const u32 n = items.end - items.off;
    if (n > NT * kWideEpt || n == 0) {  // classification and kernel disagree: record and skip
      if (threadIdx.x == 0) dev_fail(b.err, DEV_ERR_INTERNAL, items.v, n, NT);
      __syncthreads();
      items.tell();
      __syncthreads();
      items.vertex();
      items.offsets();
    } else {
      u32 at = 0;
      asm volatile("" : "+r"(at));
      build_list_wide<NT>(items.v, items.off, n, b.wgt + items.off, b.slots, b.valid, reinterpret_cast<WideShared<NT>*>(smem + at), b.err,
                          items);
    }
    if (!items.more) return;
    __syncthreads();  // the words are reused by the next list
    items.advance();
  }
}

// How many CTAs build a list of 16385 to 65536 weights together: as many as there are for each of `count` lists, three an SM.
// Builds of so many lists of 20,000 / 50,000 weights, us, with one CTA of 1024 threads a list beyond 55 of them before:
//   60 (fours)    72 / 142 -> 44 / 73; by eights, most of which have one list and some two, 55 / 81
//   180 (pairs)   121 / 275 -> 71 / 176; by eights 129 / 235
//   222 (pairs)   123 / 279 -> 77 / 186; by single CTAs 131 / 323
//   300 (single)  173 / 416 -> 131 / 314
__host__ __device__ __forceinline__ u32 long_team(u32 count, u32 ctas) {
  u32 team = kLongTeam;
  while (team > 1 && count > ctas / team) team /= 2;
  return team;
}
// A few lists more than there are pairs: the pairs take as many as they are and larger teams the rest, since a CTA alone takes
// longer than both one after the other.  So many lists of 33,000 / 63,000 weights, us, by single CTAs and this way (by CTAs of
// 1024 threads, two waves of them, it was 216 to 235 / 370 to 402):
//   223   228 / 404 -> 169 / 270          260   233 / 405 -> 180 / 299          278   234 / 408 -> 180 / 320
struct LongPlan {
  u32 team, lists;  // the first so many lists are for teams of this size,
  u32 rest;         // the others for these
};
__host__ __device__ __forceinline__ LongPlan long_plan(u32 count, u32 ctas) {
  const u32 pairs = ctas / 2;
  if (count > pairs && count <= pairs + ctas / 6) return LongPlan{2, pairs, long_team(count - pairs, ctas)};
  return LongPlan{long_team(count, ctas), 0xFFFFFFFFu, 0};
}
// More than 16384 weights, by teams of CL CTAs: those of up to 65536 (class h) if they are for teams of this size, the longer
// ones (class g) if there are eight.  Each team has a slab of scratch for up to cap weights (cap even), 12 bytes each.
// expected: how many lists of class h the host counts on, all of the graph's (whole) or at most so many.  Every number of them
// is built, also one that the host does not expect: the team size follows from what decided on the launches.
template <u32 CL>
__global__ void __launch_bounds__(kLongThreads, 3) __cluster_dims__(CL, 1, 1)
    build_long_kernel(const u32* __restrict__ list_g, const u32* __restrict__ list_h, u32* __restrict__ cls, int g, int h,
                      const __grid_constant__ ListBuild b, unsigned char* __restrict__ scratch, u64 cap, u32 ctas, u32 expected,
                      bool whole) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ u32 s_it;
  const u32 rank = blockIdx.x % CL, team = blockIdx.x / CL;
  u64* A = reinterpret_cast<u64*>(scratch + team * cap * 12);
  const LongPlan plan = long_plan(whole ? expected : min(cls[h], expected), ctas);
  const u32 all_h = cls[h], first_h = CL == plan.rest ? min(all_h, plan.lists) : 0u;
  const u32 count_g = CL == kLongTeam ? cls[g] : 0u;
  const u32 count_h = CL == plan.rest ? all_h - first_h : CL == plan.team ? min(all_h, plan.lists) : 0u;
  // Teams of several have a list each, or little more; single CTAs many, and they start when there is room.
  for (u32 it = team;; it += gridDim.x / CL) {
    if constexpr (CL == 1) {
      if (count_h == 0) break;
      if (threadIdx.x == 0) s_it = atomicAdd(cls + K_CLASSES + h, 1u);
      __syncthreads();
      it = s_it;
      __syncthreads();
    }
    if (it >= count_g + count_h) break;
    const u32 v = it < count_g ? list_g[it] : list_h[first_h + it - count_g];
    const u32 off = b.xadj[v], n = b.xadj[v + 1] - off;
    if (n > cap || n == 0) {
      if (rank == 0 && threadIdx.x == 0) dev_fail(b.err, DEV_ERR_CAPACITY, v, n, (u32)cap);
    } else {
      build_list_long<CL>(rank, v, off, n, b.wgt + off, b.slots, b.valid, reinterpret_cast<LongShared*>(smem), A,
                          reinterpret_cast<u32*>(A + cap), b.err);
    }
    cluster_sync<CL>();  // the CTAs read one another's shared memory
  }
}

// ------------------------------------------------------------------ one CTA per vertex -----
template <int T>
__device__ __forceinline__ u64 block_sum(u64 x, u64* s_red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
  __syncthreads();  // s_red may still be read from the previous reduction
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = x;
  __syncthreads();
  u64 t = 0;
#pragma unroll
  for (int w = 0; w < T / 32; ++w) t += s_red[w];
  return t;
}
template <int T>
__device__ __forceinline__ float block_max(float x, float* s_red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xFFFFFFFFu, x, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = x;
  __syncthreads();
  float t = 0.0f;
#pragma unroll
  for (int w = 0; w < T / 32; ++w) t = fmaxf(t, s_red[w]);
  return t;
}

// First index in [0, n) with a[i] >= t (a non-decreasing); n when there is none.
template <typename V>
__device__ __forceinline__ u32 lower_bound_dev(const V* a, u32 n, V t) {
  u32 lo = 0, hi = n;
  while (lo < hi) {
    const u32 mid = lo + ((hi - lo) >> 1);
    if (a[mid] < t) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Builds the table of one vertex with T threads.  D, X (u64) and LR (u32) hold n entries each,
// in shared memory or in a global slab.
template <int T>
__device__ void build_vertex_cta(u32 v, u32 off, u32 n, const float* __restrict__ wgt,
                                 Slot* __restrict__ slots, uint8_t* __restrict__ valid, u64* D,
                                 u64* X, u32* LR, u64* s_red, u32* err) {
  const u32 tid = threadIdx.x;
  const float* w = wgt + off;
  float wmax = 0.0f;
  for (u32 i = tid; i < n; i += T) wmax = fmaxf(wmax, sane_weight(__ldg(w + i)));
  wmax = block_max<T>(wmax, reinterpret_cast<float*>(s_red));
  if (!(wmax > 0.0f)) {
    for (u32 i = tid; i < n; i += T) slots[(u64)off + i] = Slot{-1.0f, i};
    if (tid == 0) valid[v] = 0;
    return;
  }
  const int B = bucket_bits(n);
  const u64 C = (u64)1 << B;
  const double scale = weight_scale(wmax, B);
  u64 acc = 0;
  for (u32 i = tid; i < n; i += T) acc += quantise(sane_weight(__ldg(w + i)), scale);
  const u64 W = block_sum<T>(acc, s_red);
  const double K = mass_factor(n, B, W);
  const u64 nC = (u64)n << B;

  // tile-wise inclusive scans: first the quantised weights (-> masses), then deficit, excess and
  // large count
  __shared__ u64 s_wq[T / 32], s_wd[T / 32], s_wx[T / 32];
  __shared__ u32 s_wl[T / 32];
  __shared__ u64 s_cq, s_cd, s_cx;
  __shared__ u32 s_cl;
  if (tid == 0) {
    s_cq = 0;
    s_cd = 0;
    s_cx = 0;
    s_cl = 0;
  }
  __syncthreads();
  const u32 lane = tid & 31, warp = tid >> 5;
  for (u32 t0 = 0; t0 < n; t0 += T) {
    const u32 i = t0 + tid;
    const u64 q = i < n ? quantise(sane_weight(__ldg(w + i)), scale) : 0;
    u64 Qi = q;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 tq = __shfl_up_sync(0xFFFFFFFFu, Qi, o);
      if (lane >= (u32)o) Qi += tq;
    }
    if (lane == 31) s_wq[warp] = Qi;
    __syncthreads();
    u64 bq = s_cq;
    for (u32 ww = 0; ww < warp; ++ww) bq += s_wq[ww];
    Qi += bq;
    u64 d = 0, x = 0;
    u32 l = 0;
    if (i < n) {
      const u64 m = cum_mass(Qi, W, nC, K) - cum_mass(Qi - q, W, nC, K);
      if (m < C) d = C - m;
      else {
        x = m - C;
        l = 1;
      }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 td = __shfl_up_sync(0xFFFFFFFFu, d, o);
      const u64 tx = __shfl_up_sync(0xFFFFFFFFu, x, o);
      const u32 tl = __shfl_up_sync(0xFFFFFFFFu, l, o);
      if (lane >= (u32)o) {
        d += td;
        x += tx;
        l += tl;
      }
    }
    if (lane == 31) {
      s_wd[warp] = d;
      s_wx[warp] = x;
      s_wl[warp] = l;
    }
    __syncthreads();
    u64 bd = s_cd, bx = s_cx;
    u32 bl = s_cl;
    for (u32 ww = 0; ww < warp; ++ww) {
      bd += s_wd[ww];
      bx += s_wx[ww];
      bl += s_wl[ww];
    }
    if (i < n) {
      D[i] = d + bd;
      X[i] = x + bx;
      LR[i] = l + bl;
    }
    __syncthreads();
    if (tid == T - 1) {
      s_cq = Qi;
      s_cd = d + bd;
      s_cx = x + bx;
      s_cl = l + bl;
    }
    __syncthreads();
  }

  for (u32 i = tid; i < n; i += T) {
    const u64 Di = D[i], Xi = X[i];
    const u64 Dp = i ? D[i - 1] : 0;
    const u32 Li = LR[i], Lp = i ? LR[i - 1] : 0;
    Slot out;
    if (Li == Lp) {  // small
      const u64 d = Di - Dp;
      u32 p = Dp ? lower_bound_dev<u64>(X, n, Dp) : lower_bound_dev<u32>(LR, n, 1u);
      if (p >= n) {
        dev_fail(err, DEV_ERR_INTERNAL, v, i, 3);
        p = i;
      }
      out.alias = p;
      out.prob = mass_to_prob(C - d, B);
    } else {
      const u32 S = lower_bound_dev<u64>(D, n, Xi + 1);
      if (S >= n) {
        out.prob = 1.0f;
        out.alias = i;
      } else {
        u32 nx = lower_bound_dev<u32>(LR, n, Li + 1);
        if (nx >= n) {
          dev_fail(err, DEV_ERR_INTERNAL, v, i, 4);
          nx = i;
        }
        out.alias = nx;
        out.prob = mass_to_prob(Xi + C - D[S], B);
      }
    }
    slots[(u64)off + i] = out;
  }
  if (tid == 0) valid[v] = 1;
}

// (A capture holds neither: an event from outside may not be waited for in it, nor one of its own outside.)
int builders_begin(skw_ctx* ctx) {
  if (ctx->tables_queued && !capturing(ctx)) SKW_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->tables_used, 0));
  return SKW_OK;
}
int builders_queued(skw_ctx* ctx) {
  if (capturing(ctx)) return SKW_OK;
  SKW_CUDA(ctx, cudaEventRecord(ctx->tables_used, ctx->stream));
  ctx->tables_queued = true;
  return SKW_OK;
}

// Zero class counters for one build.  A graph that is being captured brings its own clearing along, and has a set that no
// other build takes.
static int class_counters(skw_ctx* ctx, u32** cls) {
  constexpr unsigned kWords = skw_ctx::kClassWords, kLast = skw_ctx::kClassSets - 1;
  if (capturing(ctx)) {
    *cls = ctx->cls_counts + kLast * kWords;
    SKW_CUDA(ctx, cudaMemsetAsync(*cls, 0, kWords * sizeof(u32), ctx->stream));
    return SKW_OK;
  }
  if (ctx->cls_used == kLast) {
    SKW_CUDA(ctx, cudaMemsetAsync(ctx->cls_counts, 0, kLast * kWords * sizeof(u32), ctx->stream));
    ctx->cls_used = 0;
  }
  *cls = ctx->cls_counts + kWords * ctx->cls_used++;
  return SKW_OK;
}

// Scratch of the lists beyond 16384 weights: a slab with room for the longest for each team of eight, fewer of them when a
// giant hub would make the slabs exceed 4 GB in total, but eight at least; then, if smaller teams may be used, as much as the
// smallest need (349 MB where there are lists of 65536).  Without memory for that the teams of eight build all of them.
struct LongScratch {
  uint64_t cap = 0, cap_small = 0;  // entries of 12 bytes
  unsigned teams = 0, small = 0;
  uint64_t bytes() const { return (cap * teams + cap_small * small) * 12; }
};
// The number of lists that decides on the teams.
static u32 long_lists(const skw_ctx* ctx) { return ctx->scratch_short ? 0 : ctx->long_lists; }
static LongScratch long_scratch(const skw_ctx* ctx) {
  LongScratch s;
  if (ctx->max_degree > kHugeSmemMax) {
    s.cap = ((uint64_t)ctx->max_degree + 1) & ~1ull;
    s.teams = (unsigned)std::min<uint64_t>(ctx->sm_count * 3 / kLongTeam, std::max<uint64_t>((4ull << 30) / (s.cap * 12), 8));
    s.cap_small = std::min<uint64_t>(s.cap, kAloneMax);
    s.small = long_team(long_lists(ctx), ctx->sm_count * 3) < kLongTeam ? ctx->sm_count * 3 : 0;
  }
  return s;
}
static int reserve_scratch(skw_ctx* ctx) {
  const LongScratch s = long_scratch(ctx);
  if (s.bytes() == 0) return SKW_OK;
  const int rc = ensure_bytes(ctx, &ctx->cta_scratch, &ctx->cta_scratch_bytes, s.bytes());
  if (rc == SKW_OK || s.small == 0) return rc;
  ctx->scratch_short = true;
  const int less = ensure_bytes(ctx, &ctx->cta_scratch, &ctx->cta_scratch_bytes, long_scratch(ctx).bytes());
  if (less != SKW_OK) ctx->scratch_short = false;  // the next call asks for all of it again
  return less;
}

// Launch the class builders over the work lists of cls (see ClassLists) into `slots` and `valid`; whole: all vertices of the
// graph are in them.
static int launch_builders(skw_ctx* ctx, const ClassLists& lists, u32* cls, Slot* slots, uint8_t* valid, bool whole) {
  cudaStream_t st = ctx->stream;
  constexpr size_t kListSmem = kListWarps * kWarpBytes;
  static_assert(kListCtas * (kListSmem + 1024) <= 228 * 1024, "shared memory of an SM");
  constexpr size_t kWideA = sizeof(WideShared<512>), kWideB = sizeof(WideShared<1024>);
  static_assert(2 * (kWideA + 1024) <= 228 * 1024, "two CTAs an SM");
  static_assert(3 * (sizeof(LongShared) + 1024) <= 228 * 1024, "three CTAs an SM");
  static bool attr_set[64] = {false};
  if (!attr_set[ctx->device & 63]) {
#define SMEM(BYTES, ...) \
  SKW_CUDA(ctx, cudaFuncSetAttribute(__VA_ARGS__, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(BYTES)))
    SMEM(kListSmem, build_lists_kernel<true>);
    SMEM(kListSmem, build_lists_kernel<false>);
    SMEM(sizeof(LongShared), build_long_kernel<8>);
    SMEM(sizeof(LongShared), build_long_kernel<4>);
    SMEM(sizeof(LongShared), build_long_kernel<2>);
    SMEM(sizeof(LongShared), build_long_kernel<1>);
    SMEM(kWideA, build_wide_kernel<512>);
    SMEM(kWideB, build_wide_kernel<1024>);
#undef SMEM
    attr_set[ctx->device & 63] = true;
  }
  if (const int rc = reserve_scratch(ctx); rc != SKW_OK) return rc;
  // The classes are independent.  The long lists take few CTAs for long, so their kernels start first, on streams of their
  // own, and the many short ones fill in on the caller's.
  const int streams = ctx->max_degree > kHugeSmemMax ? 5 : ctx->max_degree > kMidSmemMax ? 3 : ctx->max_degree > kF64Max ? 2
                      : ctx->max_degree > kGroupMax ? 1 : 0;
  cudaStream_t s_h = ctx->bstream[3], s_a = ctx->bstream[2], s_b = ctx->bstream[1], s_c = ctx->bstream[0];
  if (streams) SKW_CUDA(ctx, cudaEventRecord(ctx->bfork, st));
  for (int i = 0; i < streams; ++i) SKW_CUDA(ctx, cudaStreamWaitEvent(ctx->bstream[i], ctx->bfork, 0));
  const ListBuild b{ctx->xadj, ctx->adjwgt, slots, valid, ctx->launch_err};
  if (ctx->max_degree > kHugeSmemMax) {
    // The sizes of the teams follow from the number of lists, which for all vertices is known here; for others it is at most
    // that, and the kernels of teams that are not the ones find so.  Fours have the slabs behind those of pairs, since both may
    // be at work.
    const LongScratch sc = long_scratch(ctx);
    const u32 ctas = ctx->sm_count * 3, expected = long_lists(ctx);
    const LongPlan plan = long_plan(expected, ctas);
    unsigned char* scratch = static_cast<unsigned char*>(ctx->cta_scratch);
    unsigned char* small = scratch + sc.cap * sc.teams * 12;
    auto wanted = [&](u32 team) {
      return whole ? team == plan.team || team == plan.rest : team == kLongTeam || team >= long_team(expected, ctas);
    };
#define LONG(CL, CTAS, SCRATCH, CAP, STREAM)                                                                                    \
  build_long_kernel<CL><<<CTAS, kLongThreads, sizeof(LongShared), STREAM>>>(lists.list[K_G], lists.list[K_H], cls, K_G, K_H, b, \
                                                                            SCRATCH, CAP, ctas, expected, whole);              \
  SKW_LAUNCHED(ctx)
    if (wanted(8) || ctx->max_degree > kAloneMax) {
      LONG(8, sc.teams * 8, scratch, sc.cap, ctx->bstream[4]);
    }
    if (wanted(4)) {
      LONG(4, ctas / 4 * 4, small + sc.cap_small * (ctas / 2) * 12, sc.cap_small, ctx->bstream[4]);
    }
    if (wanted(2)) {
      LONG(2, ctas / 2 * 2, small, sc.cap_small, s_h);
    }
    if (wanted(1)) {
      LONG(1, ctas, small, sc.cap_small, s_h);
    }
#undef LONG
  }
  if (ctx->max_degree > kMidSmemMax) {
    build_wide_kernel<1024><<<ctx->sm_count, 1024, kWideB, s_a>>>(lists.list[K_C2], cls, K_C2, b);
    SKW_LAUNCHED(ctx);
  }
  if (ctx->max_degree > kF64Max) {
    build_wide_kernel<512><<<ctx->sm_count * 2, 512, kWideA, s_b>>>(lists.list[K_C2A], cls, K_C2A, b);
    SKW_LAUNCHED(ctx);
  }
  const unsigned grid = ctx->sm_count * kListCtas;
  if (streams) {
    // The lists of a CTA are dealt out beforehand, so one that starts late, behind a long list, ends late.  With 64 K edges
    // or more for each there are up to four CTAs for every one that fits, and they start when those of 4097 to 8192 weights
    // run out (457 M edges: 4.69 -> 4.42 ms; 65 M: 1.73 -> 1.72).  With fewer edges they would pay for the start of each, and
    // for the wait (1 M edges: 49 -> 61 us).  More CTAs for the short lists cost more in starts, seven classes each, than
    // they gave (2.50 -> 2.55 ms at 226 M edges).
    const u64 waves = std::clamp<u64>((u64)ctx->E / ((u64)grid << 16), 1, 4);
    build_lists_kernel<true><<<(unsigned)(grid * waves), kListWarps * 32, kListSmem, waves > 1 && streams > 1 ? s_b : s_c>>>(lists, cls, b);
    SKW_LAUNCHED(ctx);
  }
  build_lists_kernel<false><<<grid, kListWarps * 32, kListSmem, st>>>(lists, cls, b);
  SKW_LAUNCHED(ctx);
  for (int i = 0; i < streams; ++i) {
    SKW_CUDA(ctx, cudaEventRecord(ctx->bjoin[i], ctx->bstream[i]));
    SKW_CUDA(ctx, cudaStreamWaitEvent(st, ctx->bjoin[i], 0));
  }
  return SKW_OK;
}

// ------------------------------------------------------------------ online frontier --------
// Collect the distinct vertices the live units stand on and bin them by degree class.  Unit u
// reads verts[(u / width) * cells + offs + u % width]; alive (optional) holds kAliveMark for
// units still running.  A vertex is claimed by the first unit that stamps it in the current collection.
constexpr u32 kAliveMark = 0xFFFFFFFFu;

// A tile of 1024 units is claimed and binned at a time, like the vertices of classify_kernel: one atomic a class and tile on
// the counters instead of one a class and warp, which all warps queued up for (hop 2 of 65,536 x 25, 10: 79 -> 28 us).
constexpr u32 kFrontierUnits = 4;  // per thread
__global__ void __launch_bounds__(256) frontier_collect_kernel(
    const u32* __restrict__ verts, u64 units, u32 width, u32 cells, u32 offs,
    const u32* __restrict__ alive, const u32* __restrict__ xadj, u32 V, u32* __restrict__ stamp,
    u32 round, u32* __restrict__ cls, const ClassLists lists, u32 cap, u32* __restrict__ err) {
  __shared__ u32 s_cnt[K_CLASSES], s_base[K_CLASSES];
  const u32 lane = threadIdx.x & 31;
  constexpr u32 kTile = 256 * kFrontierUnits;
  for (u64 u0 = (u64)blockIdx.x * kTile; u0 < units; u0 += (u64)gridDim.x * kTile) {
    if (threadIdx.x < K_CLASSES) s_cnt[threadIdx.x] = 0;
    u32 v[kFrontierUnits], rank[kFrontierUnits];
    int c[kFrontierUnits];
#pragma unroll
    for (u32 j = 0; j < kFrontierUnits; ++j) {
      const u64 u = u0 + j * 256 + threadIdx.x;
      v[j] = 0xFFFFFFFFu;
      if (u < units && (!alive || alive[u / width] == kAliveMark)) v[j] = verts[(u / width) * cells + offs + u % width];
    }
    // a hub stands in thousands of cells of one frontier: look before claiming, so that only the first few of them queue
    // up at its stamp word with an atomic
#pragma unroll
    for (u32 j = 0; j < kFrontierUnits; ++j) {
      c[j] = -1;
      if (v[j] == 0xFFFFFFFFu) continue;
      if (v[j] >= V) {
        dev_fail(err, DEV_ERR_INDEX, v[j], 0, 10);
        continue;
      }
      const u32 deg = __ldg(xadj + v[j] + 1) - __ldg(xadj + v[j]);
      if (deg && __ldcg(stamp + v[j]) != round) c[j] = degree_class(deg);
    }
#pragma unroll
    for (u32 j = 0; j < kFrontierUnits; ++j)
      if (c[j] >= 0 && atomicExch(&stamp[v[j]], round) == round) c[j] = -1;
    __syncthreads();
#pragma unroll
    for (u32 j = 0; j < kFrontierUnits; ++j) {
      const u32 same = __match_any_sync(0xFFFFFFFFu, c[j]);
      const int first = __ffs(same) - 1;
      u32 at = 0;
      if (c[j] >= 0 && lane == (u32)first) at = atomicAdd(&s_cnt[c[j]], (u32)__popc(same));
      rank[j] = __shfl_sync(0xFFFFFFFFu, at, first) + __popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (threadIdx.x < K_CLASSES && s_cnt[threadIdx.x]) s_base[threadIdx.x] = atomicAdd(&cls[threadIdx.x], s_cnt[threadIdx.x]);
    __syncthreads();
#pragma unroll
    for (u32 j = 0; j < kFrontierUnits; ++j) {
      if (c[j] < 0) continue;
      const u32 idx = s_base[c[j]] + rank[j];
      if (idx < cap) lists.list[c[j]][idx] = v[j];
      else dev_fail(err, DEV_ERR_CAPACITY, idx, cap, 11);
    }
    __syncthreads();
  }
}

int frontier_collect(skw_ctx* ctx, const u32* verts, u64 units, u32 width, u32 cells, u32 offs,
                     const u32* alive_lengths, bool new_round) {
  if (units > 0xFFFFFFFFull) return fail(ctx, SKW_ERR_ARG, "frontier of %llu units is too large",
                                         (unsigned long long)units);
  const u32 cap = (u32)(units < ctx->V ? units : ctx->V);
  void* p = ctx->frontier_lists;
  int rc = ensure_bytes(ctx, &p, &ctx->frontier_lists_bytes, sizeof(u32) * (size_t)K_CLASSES * (cap ? cap : 1));
  ctx->frontier_lists = static_cast<u32*>(p);
  if (rc != SKW_OK || (rc = builders_begin(ctx)) != SKW_OK) return rc;
  if (!ctx->stamp) {
    SKW_CUDA(ctx, dev_malloc(ctx, &ctx->stamp, sizeof(u32) * ((size_t)ctx->V + 1)));
    SKW_CUDA(ctx, cudaMemsetAsync(ctx->stamp, 0, sizeof(u32) * ((size_t)ctx->V + 1), ctx->stream));
    ctx->stamp_round = 0;
  }
  if (!new_round && ctx->stamp_round != 0) {
    // keep the round: vertices claimed earlier in this call are not collected (or built) again
  } else if (++ctx->stamp_round == 0) {  // wrapped: forget every old claim
    SKW_CUDA(ctx, cudaMemsetAsync(ctx->stamp, 0, sizeof(u32) * ((size_t)ctx->V + 1), ctx->stream));
    ctx->stamp_round = 1;
  }
  cudaStream_t st = ctx->stream;
  if (units) {
    u32* cls = nullptr;
    if ((rc = class_counters(ctx, &cls)) != SKW_OK) return rc;
    // the claim is a chain of dependent accesses (vertex, offsets, stamp): fill every thread slot of the GPU
    const u64 want = (units + 256 * kFrontierUnits - 1) / (256 * kFrontierUnits);
    const int grid = (int)(want < (u64)ctx->sm_count * 8 ? want : (u64)ctx->sm_count * 8);
    ClassLists lists;
    for (int k = 0; k < K_CLASSES; ++k) lists.list[k] = ctx->frontier_lists + (size_t)k * cap;
    frontier_collect_kernel<<<grid, 256, 0, st>>>(verts, units, width, cells, offs, alive_lengths,
                                                  ctx->xadj, ctx->V, ctx->stamp, ctx->stamp_round,
                                                  cls, lists, cap, ctx->launch_err);
    SKW_LAUNCHED(ctx);
    rc = launch_builders(ctx, lists, cls, ctx->slots, ctx->valid, false);
    if (rc != SKW_OK) return rc;
  }
  return SKW_OK;
}

}  // namespace skw

using namespace skw;

// Self-test of the bounded wait: an mbarrier that nothing ever signals.  The kernel must give up
// after its poll limit, record DEV_ERR_WAIT and return normally.
__global__ void selftest_wait_kernel(u32 limit, u32* err) {
  __shared__ __align__(8) u64 bar;
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  const bool done = mbar_wait(&bar, 0, limit);
  if (!__syncthreads_and(done ? 1 : 0) && threadIdx.x == 0) dev_fail(err, DEV_ERR_WAIT, limit, 0, 99);
}

extern "C" int skw_selftest_bounded_wait(skw_ctx* ctx) {
  if (!ctx) return SKW_ERR_ARG;
  DeviceGuard g(ctx->device);
  int rc = err_reset(ctx);
  if (rc != SKW_OK) return rc;
  selftest_wait_kernel<<<1, 64, 0, ctx->stream>>>(1u << 10, ctx->d_err);
  SKW_LAUNCHED(ctx);
  return err_check(ctx, "skw_selftest_bounded_wait");
}

namespace skw {
// Words of the work lists of `vertices` vertices; at: where the list of each class starts.
static u64 worklist_words(const skw_ctx* ctx, u32 vertices, u64* at) {
  u64 words = 0;
  for (int k = 0; k < K_CLASSES; ++k) {
    at[k] = words;
    words += class_room(k, vertices, ctx->E);
  }
  return words;
}

int reserve_builders(skw_ctx* ctx, u32 vertices) {
  u64 at[K_CLASSES];
  void* wl = ctx->worklist;
  const int rc = ensure_bytes(ctx, &wl, &ctx->worklist_cap, sizeof(u32) * worklist_words(ctx, vertices, at));
  ctx->worklist = static_cast<u32*>(wl);
  return rc != SKW_OK ? rc : reserve_scratch(ctx);
}

// Queue the construction of the tables of vertices [v_begin, v_end) into `slots` and `valid`.
int enqueue_tables(skw_ctx* ctx, u32 v_begin, u32 v_end, Slot* slots, uint8_t* valid) {
  if (v_end <= v_begin) return SKW_OK;
  int rc = reserve_builders(ctx, v_end - v_begin);
  if (rc != SKW_OK || (rc = builders_begin(ctx)) != SKW_OK) return rc;
  u64 at[K_CLASSES];
  worklist_words(ctx, v_end - v_begin, at);
  ClassLists lists;
  for (int k = 0; k < K_CLASSES; ++k) lists.list[k] = ctx->worklist + at[k];
  u32* cls = nullptr;
  if ((rc = class_counters(ctx, &cls)) != SKW_OK) return rc;
  const u64 tiles = ((u64)(v_end - v_begin) + 256 * kClassifyVertices - 1) / (256 * kClassifyVertices);
  classify_kernel<<<(unsigned)std::min<u64>(tiles, (u64)ctx->sm_count * 8), 256, 0, ctx->stream>>>(
      ctx->xadj, v_begin, v_end, cls, lists, valid);
  SKW_LAUNCHED(ctx);
  return launch_builders(ctx, lists, cls, slots, valid, v_begin == 0 && v_end == ctx->V);
}
}  // namespace skw

extern "C" int skw_alias_build_offline(skw_ctx* ctx, uint32_t v_begin, uint32_t v_end, float* ms) {
  if (!ctx) return SKW_ERR_ARG;
  if (!ctx->xadj) return fail(ctx, SKW_ERR_STATE, "skw_alias_build_offline: no graph resident");
  if (!ctx->adjwgt) return fail(ctx, SKW_ERR_STATE, "skw_alias_build_offline: weights were released");
  if (v_begin > v_end || v_end > ctx->V)
    return fail(ctx, SKW_ERR_ARG, "skw_alias_build_offline: vertex range [%u,%u) outside [0,%u]",
                v_begin, v_end, ctx->V);
  DeviceGuard g(ctx->device);
  // Records derived from the old table are no longer valid, but their memory (32 bytes an edge, four times
  // the table) stays: a rebuilt table mostly gets its records rebuilt, and freeing and allocating them again
  // took 4 to 20 ms a rebuild at 67 M edges, against 1.7 ms for everything the GPU does.  skw_walk_records_free
  // returns the memory, and so does any allocation of the context that would fail without it (dev_malloc).
  ctx->records_ready = false;
  const bool whole = v_begin == 0 && v_end == ctx->V;
  int rc = settle_queued(ctx);
  if (rc != SKW_OK) return rc;
  if ((rc = alloc_table(ctx, whole ? TableUse::kAll : TableUse::kSome)) != SKW_OK) return rc;
  rc = err_reset(ctx);
  if (rc != SKW_OK) return rc;
  cudaStream_t st = ctx->stream;
  SKW_CUDA(ctx, cudaEventRecord(ctx->ev0, st));
  if ((rc = enqueue_tables(ctx, v_begin, v_end, ctx->slots, ctx->valid)) != SKW_OK) return rc;
  SKW_CUDA(ctx, cudaEventRecord(ctx->ev1, st));
  if ((rc = err_check(ctx, "skw_alias_build_offline")) != SKW_OK) return rc;
  if (ms) SKW_CUDA(ctx, cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1));
  ctx->table_ready = ctx->slots_marked = true;
  return SKW_OK;
}

// ------------------------------------------------------------------ allocation-free variant --
// skw_alias_build_list_static: the table of ONE weight list, for hosts that must not allocate
// device memory at the time of the call.  Two kinds of caller are meant: a sampler plugged into a
// process whose framework reserved the whole HBM for its own pooling allocator at start-up (a raw
// cudaMalloc from a plug-in then fails, or takes memory behind the pool's back), and a serving
// loop that cannot afford the device-wide synchronisation cudaMalloc / cudaFree imply on its
// request path.  The prefix arrays the CTA builder needs (20 bytes per edge) therefore live in a
// fixed array inside the library image instead of a slab allocated on demand.
namespace skw {

constexpr u32 kStaticMaxDegree = 131072;  // longest weight list the static scratch holds
constexpr size_t kStaticHeader = 256;     // error record, kept apart from the arrays
// 256 B + 131072 * 20 B = 2,621,696 bytes of device memory on every GPU that loads the library,
// held until the process exits.
static __device__ __align__(256) unsigned char g_static_scratch[kStaticHeader + (size_t)kStaticMaxDegree * 20];

// The tile-wise CTA construction (build_vertex_cta) for the single list wgt[0..n), with the prefix arrays
// at `scratch` (the device address of g_static_scratch, looked up by the host).
__global__ void __launch_bounds__(1024) build_list_static_kernel(const float* __restrict__ wgt, u32 n,
                                                                 Slot* __restrict__ slots,
                                                                 uint8_t* __restrict__ valid,
                                                                 unsigned char* __restrict__ scratch) {
  __shared__ u64 s_red[1024 / 32];
  u32* err = reinterpret_cast<u32*>(scratch);
  u64* D = reinterpret_cast<u64*>(scratch + kStaticHeader);
  u64* X = D + kStaticMaxDegree;
  u32* LR = reinterpret_cast<u32*>(X + kStaticMaxDegree);
  build_vertex_cta<1024>(0, 0, n, wgt, slots, valid, D, X, LR, s_red, err);
}

static std::mutex g_static_mu;
static unsigned char* g_static_ptr[64] = {nullptr};  // device address of the array, per device

static int static_fail(char* buf, size_t len, int code, const char* fmt, ...) {
  if (buf && len) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, len, fmt, ap);
    va_end(ap);
  }
  return code;
}

}  // namespace skw

extern "C" int skw_alias_build_list_static(const float* d_weights, uint32_t n, void* d_slots,
                                           uint8_t* d_valid, void* cuda_stream, char* errbuf,
                                           size_t errbuf_len) {
  if (errbuf && errbuf_len) errbuf[0] = 0;
  if (!d_weights || !d_slots || !d_valid)
    return static_fail(errbuf, errbuf_len, SKW_ERR_ARG, "skw_alias_build_list_static: null buffer");
  if (n == 0) return static_fail(errbuf, errbuf_len, SKW_ERR_ARG, "skw_alias_build_list_static: empty weight list");
  if (n > kStaticMaxDegree)
    return static_fail(errbuf, errbuf_len, SKW_ERR_ARG,
                       "skw_alias_build_list_static: %u weights exceed the static scratch, which holds %u "
                       "(use skw_alias_build_offline for longer lists)", n, kStaticMaxDegree);
  if ((reinterpret_cast<uintptr_t>(d_slots) & 7u) || (reinterpret_cast<uintptr_t>(d_weights) & 3u))
    return static_fail(errbuf, errbuf_len, SKW_ERR_ARG, "skw_alias_build_list_static: misaligned buffer");
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess)
    return static_fail(errbuf, errbuf_len, SKW_ERR_CUDA, "skw_alias_build_list_static: cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= 64)
    return static_fail(errbuf, errbuf_len, SKW_ERR_ARG, "skw_alias_build_list_static: device %d not supported", dev);
  // a host or peer pointer handed to the kernel would fault: all three buffers must be device memory
  // of the current device
  const void* bufs[3] = {d_weights, d_slots, d_valid};
  const char* names[3] = {"d_weights", "d_slots", "d_valid"};
  for (int i = 0; i < 3; ++i) {
    cudaPointerAttributes at;
    e = cudaPointerGetAttributes(&at, bufs[i]);
    if (e != cudaSuccess || at.type != cudaMemoryTypeDevice || at.device != dev) {
      cudaGetLastError();
      return static_fail(errbuf, errbuf_len, SKW_ERR_ARG,
                         "skw_alias_build_list_static: %s is not device memory of the current device %d", names[i], dev);
    }
  }
  unsigned char* scratch = nullptr;
  {
    // First call on this device: ask the runtime where the array lives on it.  The array's name is
    // only a host-side handle; the kernel must be given this looked-up address.
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_ptr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_static_scratch);
      if (e != cudaSuccess || !p)
        return static_fail(errbuf, errbuf_len, SKW_ERR_CUDA, "skw_alias_build_list_static: cudaGetSymbolAddress: %s",
                           cudaGetErrorString(e));
      g_static_ptr[dev] = static_cast<unsigned char*>(p);
    }
    scratch = g_static_ptr[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  // the error record must start at zero; the prefix arrays are fully rewritten before they are read
  e = cudaMemsetAsync(scratch, 0, kStaticHeader, st);
  if (e != cudaSuccess)
    return static_fail(errbuf, errbuf_len, SKW_ERR_CUDA, "skw_alias_build_list_static: cudaMemsetAsync: %s", cudaGetErrorString(e));
  build_list_static_kernel<<<1, 1024, 0, st>>>(d_weights, n, static_cast<Slot*>(d_slots), d_valid, scratch);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return static_fail(errbuf, errbuf_len, SKW_ERR_CUDA, "skw_alias_build_list_static: launch: %s", cudaGetErrorString(e));
  uint32_t rec[4] = {0, 0, 0, 0};
  e = cudaMemcpyAsync(rec, scratch, sizeof rec, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess)
    return static_fail(errbuf, errbuf_len, SKW_ERR_CUDA, "skw_alias_build_list_static: %s", cudaGetErrorString(e));
  if (rec[0] != DEV_OK)
    return static_fail(errbuf, errbuf_len, SKW_ERR_DEVICE,
                       "skw_alias_build_list_static: device error %u, detail %u %u %u", rec[0], rec[1], rec[2], rec[3]);
  return SKW_OK;
}

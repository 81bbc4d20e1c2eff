// Random-walk step kernels (DeepWalk / PPR / node2vec), offline and online.
//
// Offline: takes over OfflineWalk and sample_kernel_static (src/offline_walk.cu:75-124, 181-230
// of the reference).  One lane carries one walker at a time through all of its steps and picks
// up the next walker of its stride when the current one ends, so lanes stay busy when PPR walks
// stop early; a step is: two offsets, one 8-byte {prob, alias} slot, one neighbour id, one path
// store.  Online: takes over OnlineWalkShMem / OnlineWalkKernel (src/online_walk.cu:82-166,
// 245-327), in one of two ways with identical walks: every walker computes the slot it draws
// straight from the weights (skw_walk_direct.cu), or at every step the tables of the vertices the
// live walkers stand on are built (once per distinct vertex of the frontier, by the degree-bucketed
// builders of skw_alias_build.cu) and every walker draws from the table of its vertex.
//
// Randomness: Philox4x32-10, counter (walker id low, high, step, trial), key seed ^ TAG_WALK;
// word x -> column (multiply-high by the degree), y -> acceptance uniform, z -> PPR stop test,
// w -> node2vec rejection uniform.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include <cuda.h>

#include <cub/device/device_scan.cuh>
#include <cub/iterator/transform_input_iterator.cuh>

#include "skw_ctx.h"
#include "skw_hostpool.h"
#include "skw_walk_common.cuh"

namespace skw {

int frontier_collect(skw_ctx* ctx, const u32* verts, u64 units, u32 width, u32 cells, u32 offs,
                     const u32* alive_lengths, bool new_round);

// One edge list of the CSR: its first edge and its length.
struct EdgeList {
  u32 off, deg;
};
__device__ __forceinline__ EdgeList edge_list(const WalkArgs& a, u32 v) {
  const u32 off = __ldg(a.xadj + v);
  return EdgeList{off, __ldg(a.xadj + v + 1) - off};
}

// The neighbour that random words r draw from the list of `cur`.  Returns false when there is none.  AHEAD: the neighbour of the
// drawn column is fetched beside its slot, since the draw mostly keeps it.
template <bool AHEAD>
__device__ __forceinline__ bool walk_draw(const WalkArgs& a, u32 cur, EdgeList here, Rand4 r, u32& next) {
  const u32 col = __umulhi(r.x, here.deg);
  u32 cand = col;
  if (AHEAD) next = ldg_once(a.adjncy + (u64)here.off + col);
  if (!a.unbiased) {
    const Slot s = load_slot(a.slots + (u64)here.off + col);
    if (s.prob < 0.0f) return false;  // vertex without usable weight
    cand = u01(r.y) < s.prob ? col : s.alias;
    if (cand >= here.deg) {  // a table that does not belong to this graph
      dev_fail(a.err, DEV_ERR_INDEX, cur, cand, 20);
      return false;
    }
  }
  if (!AHEAD || cand != col) next = ldg_once(a.adjncy + (u64)here.off + cand);
  return true;
}

// One step of one walker standing on `cur`.  Returns false when the walk ends here.
// r: the random words of (walker, step, trial 0).
template <int APP, bool AHEAD>
__device__ __forceinline__ bool walk_step(const WalkArgs& a, u32 step, u64 gw, u32 cur, u32& next, Rand4 r) {
  if (APP == SKW_APP_PPR && u01(r.z) < a.tp) return false;
  if (cur >= a.V) {
    dev_fail(a.err, DEV_ERR_INDEX, cur, step, (u32)gw);
    return false;
  }
  const EdgeList here = edge_list(a, cur);
  return here.deg != 0 && walk_draw<AHEAD>(a, cur, here, r, next);
}

// The same for node2vec, which also needs the list of the vertex it came from (there, deg 0 on the first
// step).  A step is a chain of dependent accesses -- slot, neighbour, search of that list -- so the list of
// the proposed vertex is fetched beside the search instead of at the start of the next step, and the list
// of the vertex that is left is handed on.
template <bool HALVING>
__device__ __forceinline__ bool walk_step_n2v(const WalkArgs& a, u32 step, u64 gw, u32 cur, u32 prev, EdgeList here,
                                              EdgeList there, u32& next, EdgeList& next_list, Rand4 r) {
  if (here.deg == 0) return false;
  for (u32 trial = 0;;) {
    if (!walk_draw<false>(a, cur, here, r, next)) return false;
    if (next >= a.V) {
      dev_fail(a.err, DEV_ERR_INDEX, next, step, (u32)gw);
      return false;
    }
    next_list = edge_list(a, next);
    if (prev == kNoVertex || n2v_keep(__fmul_rn(u01(r.w), a.fmax), next == prev, a.inv_p, a.inv_q,
                                      [&] {
                                        return HALVING ? connected_by_halving(a.adjncy, there.off, there.off + there.deg, next)
                                                       : connected(a.adjncy, there.off, there.off + there.deg, next, a.V);
                                      }))
      return true;
    if (++trial == kN2vMaxTrials) return true;  // keep the last proposal
    r = philox_tagged(a.seed, TAG_WALK, gw, step, trial);
  }
}

// Launch of the all-steps walk kernels.  A walk is a chain of dependent accesses and a warp goes on when the last of its
// lanes has its data, so a batch that leaves the GPU room takes fewer walkers a warp: as few as give `warps` warps an SM
// (what is resident: with more, the second wave costs the gain many times over).  Slots, three accesses a step, R-MAT 22,
// 80 steps: 4,096 walkers 164 -> 110 us with one walker a warp, 16,384 150 -> 127 with four, 40,000 160 -> 141 with
// eight; records, one access a step: 4,096 43 -> 38 with eight, and fewer gain no more.
// Where tables and lists take up to 8 MB the accesses are short and the warps share the issue slots: half as many warps an
// SM then (DeepWalk with uniform draws, R-MAT 14 to 16, 4,000 to 30,000 walkers: 85 -> 68 us, which 32 walkers a warp take
// 70 for; with tables 93 -> 84 us up to R-MAT 14; from 16 MB on fewer walkers a warp win again, 151 against 157 us).
// CTAs of two warps: a CTA lives as long as its unluckiest lane, and small ones keep the SMs evenly loaded to the end (slots,
// 300,000 walkers: 714 -> 668 us).  For the same reason a lane takes one walker (PPR over slots with three a thread: 1,000
// walkers 45 -> 31 us, 100,000 122 -> 100, 1 M 338 -> 309, 2 M 558 -> 532), but for PPR of many more, where a third of the
// threads starts a third of the warps (8 M walkers: 1.35 -> 1.19 ms).
struct WalkGrid {
  u32 ctas, lanes;  // walkers a warp takes at a time
};
constexpr u32 kWalkCta = 64;
static WalkGrid walk_grid(const skw_ctx* ctx, uint32_t app, u64 n, u32 warps, u32 least) {
  u32 lanes = least;
  while (lanes < 32 && n > (u64)lanes * warps * ctx->sm_count) lanes *= 2;
  const u64 per_cta = (u64)lanes * (kWalkCta / 32) * (app == SKW_APP_PPR && n > (2u << 20) ? 3 : 1);
  return WalkGrid{(u32)std::clamp<u64>((n + per_cta - 1) / per_cta, 1, 0x7FFFFFFF), lanes};
}

// Whether a draw fetches the neighbour of its column beside the slot: an access less in the chain of most steps, and one more
// where the alias is taken.  It pays while walkers wait for memory and not for its rate.  80 steps, us, without / with:
//   PPR        4,096 walkers 40 / 39 (R-MAT 22) and 45 / 44 (power law of 226 M edges), 40,000 75 / 68 and 101 / 92;
//              1 M walkers of 20 steps on the power law 325 / 346; short walks over tables in the nearest caches take their
//              neighbours from there and lose by it: at most 10 steps on R-MAT 14 with 6 MB, 16,000 38.9 / 40.2, 39,000 40.8 /
//              42.8, 32 steps 39,000 55.6 / 57.3, but 40 steps and more, fewer walkers or larger tables 0.99 to 1.15 times as fast
//   DeepWalk   tables out of cache: 1,000 walkers 96 / 89 and 111 / 98, 16,000 129 / 114 and 132 / 122, 100,000 170 / 190 and
//              455 / 524; in cache (R-MAT 16, 4,096 walkers) 73 / 77
static bool walk_ahead(const skw_ctx* ctx, uint32_t app, u64 n, u32 hop_num, bool unbiased) {
  if (unbiased) return false;
  const bool short_cached = hop_num <= 40 && ctx->E * 12 <= (8u << 20) && n > 40ull * ctx->sm_count;
  if (app == SKW_APP_PPR) return n <= 270ull * ctx->sm_count && !short_cached;
  return n <= 110ull * ctx->sm_count && ctx->E * 12 > (64u << 20);
}

// All steps of all walkers in one launch.  The first `lanes` lanes of each warp own walkers w, w + T, w + 2T ...;
// the loop body is one step, so lanes of a warp stay converged although their walkers differ.
template <int APP, bool AHEAD>
__global__ void __launch_bounds__(kWalkCta) walk_offline_kernel(const WalkArgs a, u32 lanes) {
  const u64 T = (u64)gridDim.x * (kWalkCta / 32) * lanes;
  u64 w = ((u64)blockIdx.x * (kWalkCta / 32) + threadIdx.x / 32) * lanes + (threadIdx.x & 31);
  u64 edges = 0;
  bool have = (threadIdx.x & 31) < lanes && w < a.n;
  u32 cur = 0, step = 0;
  u32* row = nullptr;
  Rand4 r{0, 0, 0, 0};  // random words of the walker's current step
  auto begin = [&]() {
    cur = __ldg(a.starts + w);
    row = a.paths + w * a.hop_num;
    row[0] = cur;
    step = 0;
    if (APP != SKW_APP_PPR) r = philox_tagged(a.seed, TAG_WALK, a.walker_base + w * a.walker_stride, 0, 0);
  };
  if (have) begin();
  while (have) {
    u32 next = 0;
    const u64 gw = a.walker_base + w * a.walker_stride;
    // The next step's words depend on nothing the step loads: computed here, they overlap its chain
    // of dependent loads (40,000 x 80 DeepWalk on the slot table: 153 -> 145 us).  Not for PPR, whose
    // walks mostly end after a step or two: there the words computed ahead are mostly thrown away
    // (8 M walkers: 1.89 -> 1.96 ms), so each step computes its own.
    Rand4 rn{0, 0, 0, 0};
    bool go;
    if (APP == SKW_APP_PPR) {
      go = step + 1 < a.hop_num &&
           walk_step<APP, AHEAD>(a, step, gw, cur, next, philox_tagged(a.seed, TAG_WALK, gw, step, 0));
    } else {
      rn = philox_tagged(a.seed, TAG_WALK, gw, step + 1, 0);
      go = step + 1 < a.hop_num && walk_step<APP, AHEAD>(a, step, gw, cur, next, r);
    }
    if (go) {
      ++step;
      row[step] = next;
      cur = next;
      if (APP != SKW_APP_PPR) r = rn;
    } else {
      a.lengths[w] = step;
      edges += step;
      w += T;
      have = w < a.n;
      if (have) begin();
    }
  }
  add_edges(a.sum, edges);
}

// The same for DeepWalk and PPR into a matrix in pinned host memory (a.paths, a.lengths as the GPU sees them): the rows go over the bus
// while the walks are under way instead of behind them.  The bus carries a write of a sector with about as many bytes of its
// own, and single cells at a fraction of its rate.  So cells wait in shared memory, two 128-byte lines of the matrix a walker
// (rows start anywhere in a line), and every 32 steps the warp writes the line that each of its walkers has filled; when in the
// 32 steps differs from warp to warp.  Cells past a walk's end get kNoVertex.
constexpr u32 kLineCells = 32, kLineRing = 2 * kLineCells;
template <int APP, bool AHEAD>
__global__ void __launch_bounds__(kWalkCta) walk_home_kernel(const WalkArgs a, u32 lanes) {
  extern __shared__ u32 rings[];  // a ring a walker, an odd number of words apart
  const u32 lane = threadIdx.x & 31, warp = blockIdx.x * (kWalkCta / 32) + threadIdx.x / 32;
  u32* const warp_rings = rings + threadIdx.x / 32 * lanes * (kLineRing + 1);
  u32* const ring = warp_rings + lane * (kLineRing + 1);
  const u64 first = (u64)warp * lanes, w = first + lane;
  const u64 gw = a.walker_base + w * a.walker_stride;
  const bool have = lane < lanes && w < a.n;
  const u32 walkers = first < a.n ? (u32)min((u64)lanes, a.n - first) : 0;  // of the warp
  // cell c of a row is place + c words behind the beginning of the line that the row starts in
  const u32 place = (u32)((((uintptr_t)a.paths >> 2) + w * a.hop_num) & (kLineCells - 1));
  bool live = have;
  u32 cur = 0, len = 0;
  Rand4 r{0, 0, 0, 0};
  if (have) {
    cur = __ldg(a.starts + w);
    if (APP != SKW_APP_PPR) r = philox_tagged(a.seed, TAG_WALK, gw, 0, 0);
  }
  u32 sent = 0;  // the lines that `sent` cells of a row fill are written
  for (u32 step = 0; walkers && step < a.hop_num;) {
    // a line of steps at a time, but for the first, which is shorter by warp
    const u32 end = min(a.hop_num, step == 0 ? kLineCells - (warp & (kLineCells - 1)) : step + kLineCells);
    if (have) {
      for (; step < end; ++step) {
        ring[(place + step) & (kLineRing - 1)] = live ? cur : kNoVertex;
        if (live && step + 1 < a.hop_num) {
          // the words of the next step are computed beside this one's loads, but for PPR, which mostly ends (walk_offline_kernel)
          Rand4 rn{0, 0, 0, 0};
          if (APP == SKW_APP_PPR) r = philox_tagged(a.seed, TAG_WALK, gw, step, 0);
          else rn = philox_tagged(a.seed, TAG_WALK, gw, step + 1, 0);
          u32 next = 0;
          live = walk_step<APP, AHEAD>(a, step, gw, cur, next, r);
          if (live) {
            cur = next;
            ++len;
            if (APP != SKW_APP_PPR) r = rn;
          }
        }
      }
    }
    step = end;
    __syncwarp();  // every lane's cells are in its ring before other lanes read them: shuffles do not order memory
    for (u32 k = 0; k < walkers; ++k) {
      const u32 at = __shfl_sync(0xFFFFFFFFu, place, k);
      const u32 lines = (at + end + (end == a.hop_num ? kLineCells - 1 : 0)) / kLineCells;
      for (u32 j = (at + sent) / kLineCells; j < lines; ++j) {
        const u32 cell = j * kLineCells + lane - at;  // wraps in front of the row's first cell
        if (cell < end)
          a.paths[(first + k) * a.hop_num + cell] = warp_rings[k * (kLineRing + 1) + ((j * kLineCells + lane) & (kLineRing - 1))];
      }
    }
    __syncwarp();  // and they are read before the next ones take their places
    sent = end;
  }
  if (have) a.lengths[w] = len;
  add_edges(a.sum, len);
}

// node2vec over the table.  A step is a chain of dependent accesses of varying length: slot and neighbour of
// every proposal, the list of the proposed vertex, and for about half of the proposals a search of the list the
// walk came from.  With one STEP per iteration every lane of a warp waits for the one with the most rejections
// and the longest search; here an iteration is one ACCESS of whatever each lane is at (the loads of all lanes
// are issued before any is used), so a walker takes as long as its own accesses.  The neighbour of the drawn
// column is fetched beside its slot, since the draw mostly keeps it, and the words of the next proposal and of
// the next step are computed while the loads are in flight.
// Bound by the latency of dependent DRAM accesses for small batches, by the rate of random accesses for large
// ones.  On the power-law graph of 117 M undirected edges, p = 2, q = 0.5, 80 steps, 40,000 / 400,000 walkers:
// 1.18 / 6.35 ms with a step per iteration, a binary search for every proposal and offsets loaded where they are
// used; with an access per iteration and searches only where they decide (n2v_keep) 0.60 / 7.2 ms when a round
// of the search probes eight places (short chain, many accesses), 0.47 / 3.1 ms when it goes by the values
// (ListSearch).  CTAs of two warps spread small batches evenly over the SMs (0.62 ms with eight); fewer
// walkers a warp than lanes gained nothing.
constexpr u32 kN2vCta = 64;
struct Draw {
  u32 x, y, w;  // column, acceptance, rejection
};
__device__ __forceinline__ Draw n2v_draw(const WalkArgs& a, u64 gw, u32 step, u32 trial) {
  const Rand4 r = philox_tagged(a.seed, TAG_WALK, gw, step, trial);
  return Draw{r.x, r.y, r.w};
}
__global__ void __launch_bounds__(kN2vCta) walk_n2v_kernel(const WalkArgs a) {
  const u64 T = (u64)gridDim.x * blockDim.x;
  u64 w = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  u64 edges = 0;
  enum : u32 { kStart, kDraw, kNeighbour, kList, kSearch, kEnd };  // what the lane does next
  u32 at = kStart;
  u32 cur = 0, prev = kNoVertex, next = 0, cand = 0, step = 0, trial = 0;
  EdgeList here{0, 0}, there{0, 0}, next_list{0, 0};  // of the vertex stood on, the one before, the one proposed
  ListSearch find;
  const bool wide = on_sector_boundary(a.adjncy);
  bool searching = false;
  Draw r{0, 0, 0}, r_retry{0, 0, 0}, r_step{0, 0, 0};  // of this proposal, the next one, the next step
  bool live = true;
  // The vote brings the lanes together again, whatever way they took through the last iteration.
  while (__any_sync(0xFFFFFFFFu, live)) {
    if (at == kEnd) {
      a.lengths[w] = step;
      edges += step;
      w += T;
      at = kStart;
    }
    if (live && at == kStart) {
      live = w < a.n;
      if (live) {
        cur = __ldg(a.starts + w);
        a.paths[w * a.hop_num] = cur;
        prev = kNoVertex;
        step = trial = 0;
        here = EdgeList{0, 0};
        if (cur < a.V) here = edge_list(a, cur);
        else dev_fail(a.err, DEV_ERR_INDEX, cur, 0, (u32)w);
        r = n2v_draw(a, a.walker_base + w * a.walker_stride, 0, 0);
        at = a.hop_num > 1 && here.deg != 0 ? kDraw : kEnd;
      }
    }
    // one access for every lane: slot and neighbour of the drawn column, neighbour of the alias, or a pair of
    // offsets (a lane that only searches re-reads)
    if (at == kDraw) cand = __umulhi(r.x, here.deg);
    const u32* nb = a.adjncy + (u64)here.off + cand;
    const u32* p = at == kDraw && !a.unbiased ? reinterpret_cast<const u32*>(a.slots + (u64)here.off + cand)
                                              : a.xadj + next;
    u32 w0 = 0, w1 = 0, w2 = 0, found[8], sector = 0;
    if (live && at <= kNeighbour) w2 = ldg_once(nb);
    if (live && at != kNeighbour && at != kEnd) {
      w0 = ldg_once(p);
      w1 = ldg_once(p + 1);
    }
    if (searching) {
      sector = find.sector(next);
      load_sector(a.adjncy, sector, find.lo, find.hi, wide, found);
    }
    if (at == kDraw) {
      const u64 gw = a.walker_base + w * a.walker_stride;
      r_retry = n2v_draw(a, gw, step, trial + 1);
      if (trial == 0) r_step = n2v_draw(a, gw, step + 1, 0);
    }
    bool proposed = at == kNeighbour;  // whether `next` becomes known
    bool judged = false, keep = true;  // whether the proposal is decided, and how
    if (at == kDraw) {
      const float prob = __uint_as_float(w0);
      proposed = a.unbiased || u01(r.y) < prob;
      at = kNeighbour;
      if (!proposed) cand = w1;
      if (!a.unbiased && prob < 0.0f) {  // vertex without usable weight
        at = kEnd;
      } else if (cand >= here.deg) {  // a table that does not belong to this graph
        dev_fail(a.err, DEV_ERR_INDEX, cur, cand, 20);
        at = kEnd;
      }
    } else if (at == kList || at == kSearch) {
      if (at == kList) next_list = EdgeList{w0, w1 - w0};
      judged = true;
      if (searching) {
        bool hit;
        at = kSearch;
        judged = find.advance(found, sector, next, hit);
        keep = __fmul_rn(u01(r.w), a.fmax) < (hit ? 1.0f : a.inv_q);
        searching = !judged;
      }
    }
    if (proposed && at != kEnd) {
      next = w2;
      at = kList;
      if (next >= a.V) {
        dev_fail(a.err, DEV_ERR_INDEX, next, step, (u32)w);
        at = kEnd;
      } else if (prev != kNoVertex) {
        keep = n2v_keep(__fmul_rn(u01(r.w), a.fmax), next == prev, a.inv_p, a.inv_q, [&] { return searching = true; });
        find = ListSearch(there.off, there.off + there.deg, a.V);  // not empty: the walk left that vertex
        judged = !keep && !searching;
      }
    }
    if (judged) {
      if (!keep && ++trial < kN2vMaxTrials) {
        r = r_retry;
        at = kDraw;
      } else if (keep || at == kSearch) {  // out of trials: the last proposal is kept, once its list is here
        ++step;
        a.paths[w * a.hop_num + step] = next;
        prev = cur;
        cur = next;
        there = here;
        here = next_list;
        trial = 0;
        r = r_step;
        at = step + 1 < a.hop_num && here.deg != 0 ? kDraw : kEnd;
      }
    }
  }
  add_edges(a.sum, edges);
}

// node2vec over the table with a step an iteration: a third of the instructions of a walker's step, and a warp waits for
// the lane with the most rejections and the longest search.
template <bool HALVING>
__global__ void __launch_bounds__(kN2vCta) walk_n2v_steps_kernel(const WalkArgs a) {
  const u64 T = (u64)gridDim.x * blockDim.x;
  u64 w = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  u64 edges = 0;
  bool have = w < a.n;
  u32 cur = 0, prev = kNoVertex, step = 0;
  EdgeList here{0, 0}, there{0, 0};  // of the vertex stood on, and of the one before
  u32* row = nullptr;
  Rand4 r{0, 0, 0, 0};  // random words of the walker's current step
  auto begin = [&]() {
    cur = __ldg(a.starts + w);
    row = a.paths + w * a.hop_num;
    row[0] = cur;
    prev = kNoVertex;
    step = 0;
    here = EdgeList{0, 0};
    if (cur < a.V) here = edge_list(a, cur);
    else dev_fail(a.err, DEV_ERR_INDEX, cur, 0, (u32)w);
    r = philox_tagged(a.seed, TAG_WALK, a.walker_base + w * a.walker_stride, 0, 0);
  };
  if (have) begin();
  while (have) {
    u32 next = 0;
    EdgeList next_list{0, 0};
    const u64 gw = a.walker_base + w * a.walker_stride;
    const Rand4 rn = philox_tagged(a.seed, TAG_WALK, gw, step + 1, 0);
    if (step + 1 < a.hop_num && walk_step_n2v<HALVING>(a, step, gw, cur, prev, here, there, next, next_list, r)) {
      ++step;
      row[step] = next;
      prev = cur;
      cur = next;
      there = here;
      here = next_list;
      r = rn;
    } else {
      a.lengths[w] = step;
      edges += step;
      w += T;
      have = w < a.n;
      if (have) begin();
    }
  }
  add_edges(a.sum, edges);
}

// Which of them: an access an iteration where walkers wait for memory, a step an iteration where the warps wait for issue
// slots, i.e. where more walkers run than the GPU holds at a time and their accesses are short or few; with the list halved
// where several rounds of walkers follow one another over lists in cache.  An access / a step / a step and halving, us:
//   lists in cache, many walkers       power law of 0.5 M edges, 300,000 x 40: 720 / 692 / 669; R-MAT 14 of 0.23 M, 1 M x 10: 578 / 411 / 354
//   mostly dead ends, short lists      R-MAT 14 of 62,000 edges, 1,000 x 80: 197 / 156 / 175
//   uniform draws, lists in cache      R-MAT 16 of 0.96 M edges, 100,000 x 40: 254 / 195 / 220; power law of 3.5 M, 70,000: 212 / 204 / 272
//   walks of a few steps               R-MAT 20 of 16 M edges, 1 M x 10: 521 / 440 / 450; power law of 226 M, 3 M x 5: 1,289 / 981
//   few vertices                       power law of 4,000 vertices, 111,000 edges, 100,000 x 40: 415 / 290
//   some dead ends, lists in cache     R-MAT 14 to 18 of 0.2 to 4 M edges, 100,000 x 40: 285 to 303 / 226 to 245 / 235 to 274
//   none of these                      power law of 11 M edges, 100,000 x 40: 301 / 314 / 397; 10,000 x 80: 367 / 524 / 738
enum class N2vWay { kAccess, kStep, kStepHalving };
static N2vWay n2v_way(const skw_ctx* ctx, const skw_walk_params* prm, u64 n, bool unbiased) {
  const u64 sms = ctx->sm_count, V = ctx->V, ends = ctx->empty_lists;
  const bool cached = ctx->E <= (unbiased ? 8u << 20 : 4u << 20);
  if (cached && n > 1500 * sms) return N2vWay::kStepHalving;
  if (ends * 2 > V && ctx->E < V * 8) return N2vWay::kStep;
  const bool many = n > 600 * sms;
  if (cached && n > 400 * sms && (unbiased || (ends * 5 > V * 2) || (many && ends * 5 > V))) return N2vWay::kStep;
  return many && (V <= 8192 || (prm->hop_num <= 17 && n > 1000 * sms)) ? N2vWay::kStep : N2vWay::kAccess;
}

// Online mode: start of a run (row[0] = start, length = "alive").
__global__ void __launch_bounds__(256) walk_online_init_kernel(const WalkArgs a) {
  for (u64 w = (u64)blockIdx.x * blockDim.x + threadIdx.x; w < a.n; w += (u64)gridDim.x * blockDim.x) {
    a.paths[w * a.hop_num] = __ldg(a.starts + w);
    a.lengths[w] = a.hop_num > 1 ? kAlive : 0u;
  }
}

// Online mode: one step of every live walker, after the tables of the frontier were built.
template <int APP>
__global__ void __launch_bounds__(256) walk_online_step_kernel(const WalkArgs a, u32 step) {
  u64 edges = 0;
  for (u64 w = (u64)blockIdx.x * blockDim.x + threadIdx.x; w < a.n; w += (u64)gridDim.x * blockDim.x) {
    if (a.lengths[w] != kAlive) continue;
    u32* row = a.paths + w * a.hop_num;
    const u32 cur = row[step];
    u32 next = 0;
    const u64 gw = a.walker_base + w * a.walker_stride;
    const Rand4 r = philox_tagged(a.seed, TAG_WALK, gw, step, 0);
    bool go;
    if (APP == SKW_APP_NODE2VEC && cur < a.V) {
      const u32 prev = step ? row[step - 1] : kNoVertex;
      EdgeList next_list;
      go = walk_step_n2v<false>(a, step, gw, cur, prev, edge_list(a, cur), step ? edge_list(a, prev) : EdgeList{0, 0}, next,
                         next_list, r);
    } else {
      go = walk_step<APP, false>(a, step, gw, cur, next, r);
    }
    if (go) {
      row[step + 1] = next;
      if (step + 2 == a.hop_num) {
        a.lengths[w] = step + 1;
        edges += step + 1;
      }
    } else {
      a.lengths[w] = step;
      edges += step;
    }
  }
  add_edges(a.sum, edges);
}

// ------------------------------------------------------------------ fused walk records -----
// B200 has room for a wider table: one 32-byte record per edge slot that already holds both
// outcomes of the draw together with what the NEXT step needs (offset and degree of the vertex
// reached), so a step is ONE random 32-byte access (one 256-bit load) instead of three dependent
// ones (offsets -> slot -> neighbour id).  Random DRAM accesses per step, not bytes, bound the
// walk on this memory system, so this is worth 4x the table size.  The records are derived from
// the alias table and the CSR and give bit-identical walks.
//   w0 prob | w1 neighbour if kept | w2 its first-edge offset | w3 its usable degree
//           | w4 neighbour via alias | w5 its offset          | w6 its usable degree | w7 alias
// "usable degree" is 0 for a vertex without out-edges or without usable weight: the walk ends there.
struct __align__(32) WalkRecord {
  u32 w[8];
};

// One 256-bit load.  By default an L1 miss pulls the whole 128-byte line (4 sectors) from DRAM; a
// record is one sector and is used once, so ask for the smallest L2 fetch (64 bytes) and keep it
// out of L1.  Measured on B200: same access rate, half the DRAM traffic.
__device__ __forceinline__ void load_record(const WalkRecord* p, u32 (&w)[8]) {
  asm volatile("ld.global.nc.L1::no_allocate.L2::64B.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(p));
}

constexpr u32 kRecTile = 1024, kRecSpan = 1024;  // slots of a tile of the records build, offsets it keeps at hand
constexpr u32 kRecPer = 4, kRecCta = kRecTile / kRecPer;  // slots a thread

// vinfo[v] = {first-edge offset, usable degree}; vbits = one bit per vertex, set when the usable
// degree is not zero.  The bitmap is V/8 bytes and stays in L2, so a walker that starts on a dead
// end (most uniformly random starts of a directed R-MAT graph) never touches DRAM for it.
__global__ void __launch_bounds__(256) vertex_info_kernel(const u32* __restrict__ xadj,
                                                          const Slot* __restrict__ slots, u32 V,
                                                          uint2* __restrict__ vinfo, u32* __restrict__ vbits,
                                                          u32* __restrict__ unusable, u32* __restrict__ tile_first) {
  const u64 T = (u64)gridDim.x * blockDim.x;
  const u64 rounds = ((u64)V + T - 1) / T;
  for (u64 it = 0; it < rounds; ++it) {  // whole warps stay in the loop: the ballot needs them
    const u64 v = it * T + (u64)blockIdx.x * blockDim.x + threadIdx.x;
    u32 eff = 0;
    if (v < V) {
      const u32 off = xadj[v], deg = xadj[v + 1] - off;
      eff = deg;
      if (deg && load_slot(slots + off).prob < 0.0f) {
        eff = 0;
        atomicAdd(unusable, 1u);  // has out-edges but no table (all weights unusable, or not built yet): rare
      }
      vinfo[v] = make_uint2(off, eff);
      // the tiles of the records build whose first slot lies in this list
      for (u64 t = ((u64)off + kRecTile - 1) / kRecTile; t * kRecTile < (u64)off + deg; ++t) tile_first[t] = (u32)v;
    }
    const u32 word = __ballot_sync(0xFFFFFFFFu, eff != 0);
    if ((threadIdx.x & 31) == 0 && v < V) vbits[v >> 5] = word;
  }
}

// A CTA per tile of kRecTile consecutive slots, neighbouring lanes on neighbouring slots.  The vertex of a tile's first
// slot is at hand (tile_first); the offsets of the vertices of the tile are copied to shared memory (75 on average on the
// R-MAT graphs, empty ones included), where every list also marks its first slot: a warp bisects the offsets for the
// first of its 32 slots and goes by the marks from there.  A tile that spans more vertices (long runs of empty ones)
// bisects the global array for every slot.  A neighbour's {offset, degree} is a random access; the one reached through the
// alias mostly belongs to a slot of the same tile, whose thread has fetched it already.
// Bound by the pipe of L1 and shared memory (a random lookup a slot, and a record a thread takes a wavefront where a warp's
// records side by side take a quarter) and by waiting in the phases of a tile, so four slots a thread in 38 registers and 48
// warps an SM beat eight in 60 and 32: R-MAT 22, 65 M slots 845 -> 754 us, R-MAT 24, 457 M slots 7.49 -> 6.67 ms (4.1 ->
// 4.6 TB/s of DRAM).  Before: 1.10 ms with two random lookups a slot and every tile's vertices bisected from the whole offset
// array, 0.91 with a bisection per slot.  Two slots a thread and 64 warps: 755 us / 6.64 ms.  Slower: two 16-byte stores a
// record 834, halves exchanged between neighbours so that 16 records fill a store 919, records laid out in shared memory and
// copied out by the bulk engine, a tile or 32 at a time, 1569 and 1680; the next tile fetched to L2 ahead 884.
__device__ __forceinline__ u32 last_vertex_at_or_before(const u32* __restrict__ xadj, u32 lo, u32 hi, u32 e) {
  while (lo < hi) {  // last v in [lo, hi] with xadj[v] <= e
    const u32 mid = lo + ((hi - lo + 1) >> 1);
    if (__ldg(xadj + mid) <= e) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
__global__ void __launch_bounds__(kRecCta, 6) walk_records_kernel(const u32* __restrict__ xadj,
                                                              const u32* __restrict__ adjncy,
                                                              const Slot* __restrict__ slots,
                                                              const uint2* __restrict__ vinfo,
                                                              const u32* __restrict__ tile_first, u32 V, u64 E,
                                                              WalkRecord* __restrict__ rec, u32* __restrict__ err) {
  __shared__ u32 s_x[kRecSpan + 1];
  __shared__ __align__(16) u32 s_nbr[kRecTile];
  __shared__ __align__(16) uint2 s_info[kRecTile];
  __shared__ __align__(16) uint16_t s_head[kRecTile];  // place of the list that starts here, plus 1
  const u64 tiles = (E + kRecTile - 1) / kRecTile;
  for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const u64 e0 = tile * kRecTile;
    const u32 here = (u32)min((u64)kRecTile, E - e0);
    const u32 v0 = __ldg(tile_first + tile), v1 = tile + 1 < tiles ? __ldg(tile_first + tile + 1) : V - 1;
    u32 nbr[kRecPer];
    Slot sl[kRecPer];
#pragma unroll
    for (u32 k = 0; k < kRecPer; ++k) {  // (past the end: the last slot again)
      const u32 e = (u32)e0 + min(threadIdx.x + kRecCta * k, here - 1);
      sl[k] = load_slot(slots + e);
      nbr[k] = __ldg(adjncy + e);
    }
    const bool staged = v1 - v0 < kRecSpan;
    *reinterpret_cast<uint2*>(s_head + threadIdx.x * kRecPer) = make_uint2(0u, 0u);
    static_assert(kRecPer == 4, "four half-words a thread are cleared");
    __syncthreads();
    if (staged) {
      for (u32 i = threadIdx.x; i <= v1 - v0 + 1; i += kRecCta) {
        const u32 x = __ldg(xadj + v0 + i);
        s_x[i] = x;
        if (i <= v1 - v0 && x - (u32)e0 < here && __ldg(xadj + v0 + i + 1) != x) s_head[x - (u32)e0] = (uint16_t)(i + 1);
      }
    }
    uint2 info[kRecPer];
#pragma unroll
    for (u32 k = 0; k < kRecPer; ++k) {
      info[k] = make_uint2(0u, 0u);
      if (nbr[k] < V) info[k] = __ldg(vinfo + nbr[k]);
      else dev_fail(err, DEV_ERR_INDEX, (u32)e0 + min(threadIdx.x + kRecCta * k, here - 1), nbr[k], 22);
    }
#pragma unroll
    for (u32 k = 0; k < kRecPer; ++k) {
      s_nbr[threadIdx.x + kRecCta * k] = nbr[k];
      s_info[threadIdx.x + kRecCta * k] = info[k];
    }
    __syncthreads();
    // the vertex (relative to v0) of the first slot of each of the warp's runs of 32, by one lane each
    const u32 lane = threadIdx.x & 31;
    u32 first = 0;
    if (staged && lane < kRecPer) {
      const u32 e = (u32)e0 + min(threadIdx.x - lane + kRecCta * lane, here - 1);
      for (u32 hi = v1 - v0; first < hi;) {
        const u32 mid = (first + hi + 1) >> 1;
        if (s_x[mid] <= e) first = mid;
        else hi = mid - 1;
      }
    }
#pragma unroll
    for (u32 k = 0; k < kRecPer; ++k) {
      const u32 i = threadIdx.x + kRecCta * k;
      u32 v = __shfl_sync(0xFFFFFFFFu, first, k);
      const u32 head = s_head[i];
      const u32 heads = __ballot_sync(0xFFFFFFFFu, head != 0) & (0xFFFFFFFFu >> (31 - lane));  // up to this lane
      const u32 mark = __shfl_sync(0xFFFFFFFFu, head, heads ? 31 - __clz((int)heads) : 0);
      if (heads) v = mark - 1;
      if (i < here) {
        if (!staged) v = last_vertex_at_or_before(xadj, v0, v1, (u32)e0 + i) - v0;
        const u32 off = staged ? s_x[v] : __ldg(xadj + v0 + v);
        const u32 deg = (staged ? s_x[v + 1] : __ldg(xadj + v0 + v + 1)) - off;
        u32 alias = sl[k].alias;
        if (alias >= deg) {  // a table that does not belong to this graph: keep the read inside the list
          dev_fail(err, DEV_ERR_INDEX, (u32)e0 + i, alias, 22);
          alias = 0;
        }
        const u32 at = off + alias - (u32)e0;  // (wraps around below the tile)
        u32 n_alias;
        uint2 i_alias;
        if (at < here) {
          n_alias = s_nbr[at];
          i_alias = s_info[at];
        } else {
          n_alias = __ldg(adjncy + (u64)off + alias);
          i_alias = n_alias < V ? __ldg(vinfo + n_alias) : make_uint2(0u, 0u);
        }
        asm volatile("st.global.v8.u32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(rec + e0 + i), "r"(__float_as_uint(sl[k].prob)),
                     "r"(nbr[k]), "r"(info[k].x), "r"(info[k].y), "r"(n_alias), "r"(i_alias.x), "r"(i_alias.y), "r"(alias)
                     : "memory");
      }
    }
    __syncthreads();
  }
}

struct RecordWalkArgs {
  const WalkRecord* rec;
  const uint2* vinfo;
  const u32* vbits;
  const u32* starts;
  u32* paths;
  u32* heads;  // walk_records_ppr_kernel: the first cells of the rows go here, back to back, or (null) to the rows
  u32* lengths;
  unsigned long long* sum;
  u32* err;
  u64 n;
  u64 seed;
  u64 walker_base;
  u64 walker_stride;
  u32 V;
  u32 hop_num;
  float tp;
  u32 unbiased;  // uniform neighbour: the column's own neighbour is always kept (SKW_WALK_UNBIASED)
};

// Same lane-owns-a-stride loop as walk_offline_kernel; a step is one record load.
template <int APP>
__global__ void __launch_bounds__(kWalkCta) walk_records_walk_kernel(const RecordWalkArgs a, u32 lanes) {
  const u64 T = (u64)gridDim.x * (kWalkCta / 32) * lanes;
  u64 w = ((u64)blockIdx.x * (kWalkCta / 32) + threadIdx.x / 32) * lanes + (threadIdx.x & 31);
  u64 edges = 0;
  bool have = (threadIdx.x & 31) < lanes && w < a.n;
  u32 off = 0, deg = 0, step = 0;
  u32* row = nullptr;
  Rand4 r{0, 0, 0, 0};  // random words of the walker's current step
  auto begin = [&]() {
    const u32 cur = __ldg(a.starts + w);
    row = a.paths + w * a.hop_num;
    row[0] = cur;
    step = 0;
    if (cur >= a.V) {
      dev_fail(a.err, DEV_ERR_INDEX, cur, 0, (u32)w);
      off = 0;
      deg = 0;
    } else if ((__ldg(a.vbits + (cur >> 5)) >> (cur & 31)) & 1u) {
      const uint2 vi = ldg_once(a.vinfo + cur);
      off = vi.x;
      deg = vi.y;
    } else {
      off = 0;
      deg = 0;
    }
    r = philox_tagged(a.seed, TAG_WALK, a.walker_base + w * a.walker_stride, 0, 0);
  };
  if (have) begin();
  while (have) {
    bool go = step + 1 < a.hop_num && deg != 0;
    if (APP == SKW_APP_PPR && go && u01(r.z) < a.tp) go = false;
    if (go) {
      u32 rw[8];
      load_record(a.rec + (u64)off + __umulhi(r.x, deg), rw);
      // the next step's random words do not depend on the record: computing them here overlaps the
      // load's latency (what a walk is made of when few walkers are in flight)
      const Rand4 rn = philox_tagged(a.seed, TAG_WALK, a.walker_base + w * a.walker_stride, step + 1, 0);
      const bool keep = a.unbiased || u01(r.y) < __uint_as_float(rw[0]);
      ++step;
      row[step] = keep ? rw[1] : rw[4];
      off = keep ? rw[2] : rw[5];
      deg = keep ? rw[3] : rw[6];
      r = rn;
    } else {
      a.lengths[w] = step;
      edges += step;
      w += T;
      have = w < a.n;
      if (have) begin();
    }
  }
  add_edges(a.sum, edges);
}

// PPR over the walk records, one warp per chunk of kChunk consecutive walkers.
//
// Most PPR walks end after a handful of steps, so the loop is dominated by handing lanes their
// next walker.  Set-up: the chunk's start vertices and their {offset, degree} entries are fetched
// up front, independent loads issued together, and parked in per-walker staging rows in shared
// memory (cell 0 = start, cells 1, 2 = offset, degree until the walker's first steps overwrite
// them).  Lanes take walkers from a warp-wide counter (ballot + popc, no atomics) as they become
// free, which costs two shared-memory reads, so the loop holds exactly one dependent global load
// per step.  The first kStage cells of every path are staged in shared memory and written out,
// with the lengths, when the chunk is done (8 lanes per row); cells from kStage on go straight to
// the row.
//
// Measured on B200, 8 M walkers on the scale-26 graph (20.9 M sampled edges per launch): 0.97 ms
// against 1.17 ms for the lane-owns-a-stride kernel; 0.67 ms with the path stores left out, i.e.
// the 8 M isolated row prefixes (one or two 32-byte sectors each, rows hop_num * 4 bytes apart)
// cost DRAM about as much as the record reads, whether they are written step by step or together
// at the end, with default or streaming stores; padding the prefixes to whole 32-byte sectors
// (so that no partly written sector leaves L2) made the launch 12 % slower.  Chunks of 64 walkers
// with 8 warps per CTA were the best of {64, 128, 256} x {4, 8, 16}.
// A batch of 1 M walkers is 1.65 waves of resident CTAs.  Two ways of avoiding the second wave were
// built and compared with this kernel on one GPU, back to back (1 M walkers on the scale-22 graph /
// 8 M on scale 26): chunks handed out from a global atomic cursor to a persistent grid, 0.185 / 0.996 ms
// against 0.174 / 0.973 ms here; chunks of 128 walkers, so that every CTA is resident at once, 0.172 /
// 1.049 ms against 0.173 / 0.971 ms.  Neither helps: the hardware's CTA backfill already keeps the SMs
// loaded, and a small batch is bounded by its longest walks -- with tp = 0.15 the longest of a million
// walks makes 80 to 100 dependent steps, slow ones while the memory system is saturated (300 K lanes in
// flight at 43 G accesses/s are 7 us per access) and 0.6-0.9 us each once it has drained.
constexpr u32 kChunk = 64, kStage = 8;
template <int WARPS, int CHUNK, int STAGE>
__global__ void __launch_bounds__(WARPS * 32, 2048 / (WARPS * 32)) walk_records_ppr_kernel(const RecordWalkArgs a) {
  constexpr u32 kPitch = STAGE + 1;
  __shared__ u32 s_buf[WARPS][CHUNK * kPitch];
  __shared__ uint16_t s_len[WARPS][CHUNK];
  const u32 lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const u64 w_begin = ((u64)blockIdx.x * WARPS + wib) * CHUNK;
  if (w_begin >= a.n) return;  // the whole warp leaves; nothing below synchronises the CTA
  const u32 cnt = (u32)min((u64)CHUNK, a.n - w_begin);
  u32* buf = s_buf[wib];
  uint16_t* len = s_len[wib];
  {
    u32 st[CHUNK / 32];
    bool live[CHUNK / 32];
#pragma unroll
    for (int k = 0; k < (int)(CHUNK / 32); ++k) {
      const u32 i = k * 32 + lane;
      st[k] = i < cnt ? __ldg(a.starts + w_begin + i) : 0u;
    }
#pragma unroll
    for (int k = 0; k < (int)(CHUNK / 32); ++k) {
      const u32 i = k * 32 + lane;
      live[k] = false;
      if (i < cnt) {
        if (st[k] >= a.V) dev_fail(a.err, DEV_ERR_INDEX, st[k], 0, (u32)(w_begin + i));
        else live[k] = (__ldg(a.vbits + (st[k] >> 5)) >> (st[k] & 31)) & 1u;
      }
    }
#pragma unroll
    for (int k = 0; k < (int)(CHUNK / 32); ++k) {
      const u32 i = k * 32 + lane;
      uint2 vi = make_uint2(0u, 0u);
      if (live[k]) vi = ldg_once(a.vinfo + st[k]);
      if (i < cnt) {
        buf[i * kPitch] = st[k];
        buf[i * kPitch + 1] = vi.x;
        buf[i * kPitch + 2] = vi.y;
      }
    }
  }
  __syncwarp();
  const u32 lt = (1u << lane) - 1u;
  u32 next = 0;  // walkers of the chunk handed out so far (the same in every lane)
  bool active = false;
  u32 local = 0, off = 0, deg = 0, step = 0;
  u64 edges = 0;
  Rand4 r{0, 0, 0, 0};  // random words of the walker's current step
  for (;;) {
    const u32 need = __ballot_sync(0xFFFFFFFFu, !active);
    if (need && next < cnt) {
      const u32 mine = next + __popc(need & lt);
      if (!active && mine < cnt) {
        local = mine;
        off = buf[local * kPitch + 1];
        deg = buf[local * kPitch + 2];
        step = 0;
        active = true;
        r = philox_tagged(a.seed, TAG_WALK, a.walker_base + (w_begin + local) * a.walker_stride, 0, 0);
      }
      next = min(cnt, next + (u32)__popc(need));
    }
    if (!__any_sync(0xFFFFFFFFu, active)) break;
    if (active) {
      const bool go = step + 1 < a.hop_num && deg != 0 && !(u01(r.z) < a.tp);
      if (go) {
        u32 rw[8];
        load_record(a.rec + (u64)off + __umulhi(r.x, deg), rw);
        // the next step's random words do not depend on the record: computing them here overlaps the
        // load's latency, which is what the end of a pass is made of
        const u32 ry = r.y;
        r = philox_tagged(a.seed, TAG_WALK, a.walker_base + (w_begin + local) * a.walker_stride, step + 1, 0);
        const bool keep = a.unbiased || u01(ry) < __uint_as_float(rw[0]);
        ++step;
        const u32 nv = keep ? rw[1] : rw[4];
        if (step < (u32)STAGE) buf[local * kPitch + step] = nv;
        else a.paths[(w_begin + local) * a.hop_num + step] = nv;
        off = keep ? rw[2] : rw[5];
        deg = keep ? rw[3] : rw[6];
      } else {
        len[local] = (uint16_t)step;
        edges += step;
        active = false;
      }
    }
  }
  __syncwarp();
  // write-out: 8 lanes per row, four neighbouring rows per pass; then the lengths, coalesced
  static_assert(STAGE == 8, "a lane a cell");
  for (u32 r = lane >> 3; r < cnt; r += 4) {
    const u32 c = lane & 7;
    const u32 cells = min((u32)len[r] + 1u, (u32)STAGE);
    if (a.heads) a.heads[(w_begin + r) * STAGE + c] = buf[r * kPitch + c];  // (whole sectors)
    else if (c < cells) a.paths[(w_begin + r) * a.hop_num + c] = buf[r * kPitch + c];
  }
  for (u32 i = lane; i < cnt; i += 32) a.lengths[w_begin + i] = len[i];
  add_edges(a.sum, edges);
}

// Copy the written part of every path row (cells 0..length) from the device matrix into a host
// matrix that the GPU can address (pinned memory), 8 lanes per row.  For PPR most rows hold a
// handful of cells, so this moves a few percent of what a copy of the whole matrix would.
__global__ void __launch_bounds__(256) copy_row_prefixes_kernel(const u32* __restrict__ src,
                                                                u32* __restrict__ dst,
                                                                const u32* __restrict__ lengths, u64 n,
                                                                u32 hop_num) {
  const u32 sub = threadIdx.x & 7;
  const u64 rows_per_pass = ((u64)gridDim.x * blockDim.x) >> 3;
  for (u64 w = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 3; w < n; w += rows_per_pass) {
    const u32 cells = min(__ldg(lengths + w) + 1u, hop_num);
    const u32* s = src + w * hop_num;
    u32* d = dst + w * hop_num;
    for (u32 c = sub; c < cells; c += 8) d[c] = s[c];
  }
}

// Packed result: the written cells of row w (0..length) go to packed[offs[w] ..), rows back to
// back in walker order; 8 lanes per row, so neighbouring rows fill whole sectors of the output.
struct CellsOfRow {
  __host__ __device__ u64 operator()(u32 length) const { return (u64)length + 1; }
};

__global__ void __launch_bounds__(256) pack_rows_kernel(const u32* __restrict__ src, u32* __restrict__ packed,
                                                        const u32* __restrict__ lengths,
                                                        const u64* __restrict__ offs, u64 n, u32 hop_num,
                                                        u64 capacity, u64* __restrict__ total,
                                                        uint8_t* __restrict__ lengths8) {
  const u32 sub = threadIdx.x & 7;
  const u64 rows_per_pass = ((u64)gridDim.x * blockDim.x) >> 3;
  for (u64 w = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 3; w < n; w += rows_per_pass) {
    const u32 len = __ldg(lengths + w);
    const u32 cells = min(len + 1u, hop_num);
    const u64 o = __ldg(offs + w);
    if (lengths8 && sub == 0) lengths8[w] = (uint8_t)len;  // the caller asked for one byte per walk
    if (w == n - 1 && sub == 0) *total = o + cells;  // cells the whole batch needs
    // rows that do not fit are left out: the host compares *total with the capacity and packs again
    // into a larger buffer
    if (o + cells > capacity) continue;
    const u32* s = src + w * hop_num;
    for (u32 c = sub; c < cells; c += 8) packed[o + c] = ldg_once(s + c);
  }
}

// The same where the first kStage cells of the rows are in `heads`, back to back.  A warp takes 32 rows: lengths, places and
// then the heads of all of them are fetched with independent loads, eight lanes a row; longer rows go on with eight lanes each,
// or the whole warp where most are long.  A row at a time, each group of eight lanes waits for two dependent accesses a row:
// 667,000 PPR walks of at most 100 steps, 2.7 M cells, 46 us.
__global__ void __launch_bounds__(256) pack_heads_kernel(const u32* __restrict__ src, const u32* __restrict__ heads,
                                                        u32* __restrict__ packed, const u32* __restrict__ lengths,
                                                        const u64* __restrict__ offs, u64 n, u32 hop_num,
                                                        u64 capacity, u64* __restrict__ total,
                                                        uint8_t* __restrict__ lengths8) {
  static_assert(kStage == 8, "a lane a cell");
  const u32 lane = threadIdx.x & 31, sub = lane & 7, group = lane >> 3;
  const u64 stride = ((u64)gridDim.x * blockDim.x >> 5) * 32;
  for (u64 w0 = (((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; w0 < n; w0 += stride) {
    const u64 w = w0 + lane;
    u32 cells = 0;
    u64 o = 0;
    if (w < n) {
      const u32 len = __ldg(lengths + w);
      cells = min(len + 1u, hop_num);
      o = __ldg(offs + w);
      if (lengths8) lengths8[w] = (uint8_t)len;  // the caller asked for one byte per walk
      if (w == n - 1) *total = o + cells;        // cells the whole batch needs
      // rows that do not fit are left out: the host compares *total with the capacity and packs again
      // into a larger buffer
      if (o + cells > capacity) cells = 0;
    }
    u32 first[8];
#pragma unroll
    for (u32 r = 0; r < 8; ++r) {
      const u32 row = r * 4 + group;
      const u32 have = __shfl_sync(0xFFFFFFFFu, cells, row);
      first[r] = 0;
      if (sub < have) first[r] = __ldg(heads + (w0 + row) * kStage + sub);
    }
#pragma unroll
    for (u32 r = 0; r < 8; ++r) {
      const u32 row = r * 4 + group;
      const u32 have = __shfl_sync(0xFFFFFFFFu, cells, row);
      const u64 to = __shfl_sync(0xFFFFFFFFu, o, row);
      if (sub < have) packed[to + sub] = first[r];
    }
    u32 more = __ballot_sync(0xFFFFFFFFu, cells > 8);
    const u32 lanes = __popc(more) > 16 ? 32 : 8;  // a row
    while (more) {
      // the next row, or the next four
      u32 row = 32;
      for (u32 g = 0; more && g < 32 / lanes; ++g) {
        if (lane / lanes == g) row = __ffs(more) - 1;
        more &= more - 1;
      }
      const u32 have = __shfl_sync(0xFFFFFFFFu, cells, row & 31);
      const u64 to = __shfl_sync(0xFFFFFFFFu, o, row & 31);
      if (row < 32) {
        const u32* from = src + (w0 + row) * hop_num;
        for (u32 c = 8 + lane % lanes; c < have; c += lanes) packed[to + c] = ldg_once(from + c);
      }
    }
  }
}

__global__ void __launch_bounds__(256) generate_starts_kernel(u32* __restrict__ starts, u64 n,
                                                              u64 id_base, u64 seed, u32 V) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
    const Rand4 r = philox_tagged(seed, TAG_STRT, id_base + i, 0, 0);
    starts[i] = __umulhi(r.x, V);
  }
}

// Measurement aid: a dependent chain of random 32-byte record loads, the memory behaviour of a walk
// stripped of everything else.  Every thread follows `iters` pseudo-random hops through `nrec`
// records with the same load instruction the record walk uses.
__global__ void __launch_bounds__(256) probe_gather_kernel(const WalkRecord* __restrict__ rec, u64 nrec,
                                                           u32 iters, unsigned long long* __restrict__ sink) {
  const u64 tid = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  u64 cur = (tid * 0x9E3779B97F4A7C15ull) % nrec;
  u32 acc = 0;
  for (u32 it = 0; it < iters; ++it) {
    u32 w[8];
    load_record(rec + cur, w);
    acc += w[0];
    u64 x = cur * 31 + w[7] + it + tid;
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    cur = x % nrec;
  }
  if (acc == 0x12345677u) atomicAdd(sink, 1ull);  // keeps the loads alive
}

static int grid_for(const skw_ctx* ctx, u64 n, int per_sm) {
  const u64 want = (n + 255) / 256;
  const u64 cap = (u64)ctx->sm_count * per_sm;
  return (int)(want < cap ? (want ? want : 1) : cap);
}

}  // namespace skw

using namespace skw;

extern "C" {

int skw_generate_starts_device(skw_ctx* ctx, uint64_t n, uint64_t id_base, uint64_t seed,
                               uint32_t* d_starts) {
  if (!ctx || (n && !d_starts)) return SKW_ERR_ARG;
  if (!ctx->V) return fail(ctx, SKW_ERR_STATE, "skw_generate_starts_device: no graph resident");
  DeviceGuard g(ctx->device);
  if (n) {
    generate_starts_kernel<<<grid_for(ctx, n, 8), 256, 0, ctx->stream>>>(d_starts, n, id_base, seed, ctx->V);
    SKW_LAUNCHED(ctx);
  }
  return SKW_OK;
}

int skw_walk_records_build(skw_ctx* ctx, float* ms) {
  if (!ctx) return SKW_ERR_ARG;
  if (!ctx->table_ready) return fail(ctx, SKW_ERR_STATE, "skw_walk_records_build: build or import the alias table first");
  DeviceGuard g(ctx->device);
  if (const int rc = settle_queued(ctx); rc != SKW_OK) return rc;
  ctx->records_ready = false;
  ctx->records_building = true;
  // any failure below leaves no half-built records behind
  auto body = [&]() -> int {
    if (!ctx->records) SKW_CUDA(ctx, dev_malloc(ctx, &ctx->records, sizeof(WalkRecord) * (ctx->E ? ctx->E : 1)));
    if (!ctx->vinfo) SKW_CUDA(ctx, dev_malloc(ctx, &ctx->vinfo, sizeof(uint2) * ((size_t)ctx->V + 1)));
    // the bitmap, and behind it the first vertex of every tile of the records build
    const u64 tiles = (ctx->E + kRecTile - 1) / kRecTile;
    if (!ctx->vbits) SKW_CUDA(ctx, dev_malloc(ctx, &ctx->vbits, sizeof(u32) * ((size_t)ctx->V / 32 + 1 + tiles)));
    u32* tile_first = static_cast<u32*>(ctx->vbits) + (size_t)ctx->V / 32 + 1;
    int rc = err_reset(ctx);
    if (rc != SKW_OK) return rc;
    cudaStream_t st = ctx->stream;
    SKW_CUDA(ctx, cudaEventRecord(ctx->ev0, st));
    if (ctx->V) {
      vertex_info_kernel<<<ctx->sm_count * 16, 256, 0, st>>>(ctx->xadj, ctx->slots, ctx->V,
                                                              static_cast<uint2*>(ctx->vinfo), static_cast<u32*>(ctx->vbits),
                                                              reinterpret_cast<u32*>(ctx->d_sum + 3), tile_first);
      SKW_LAUNCHED(ctx);
    }
    if (ctx->E && ctx->V) {
      const u64 cap = (u64)ctx->sm_count * 32;
      walk_records_kernel<<<(unsigned)(tiles < cap ? tiles : cap), kRecCta, 0, st>>>(
          ctx->xadj, ctx->adjncy, ctx->slots, static_cast<const uint2*>(ctx->vinfo), tile_first, ctx->V, ctx->E,
          static_cast<WalkRecord*>(ctx->records), ctx->d_err);
      SKW_LAUNCHED(ctx);
    }
    SKW_CUDA(ctx, cudaEventRecord(ctx->ev1, st));
    if ((rc = err_check(ctx, "skw_walk_records_build")) != SKW_OK) return rc;  // synchronises the stream
    if (ms) SKW_CUDA(ctx, cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1));
    return SKW_OK;
  };
  const int rc = body();
  ctx->records_building = false;
  if (rc != SKW_OK) {
    const std::string why = ctx->err;
    cudaGetLastError();
    drop_records(ctx);
    ctx->err = why;
    return rc;
  }
  ctx->records_ready = true;
  // every vertex with out-edges has a usable table: the records' offsets and degrees are then those of
  // the graph itself, and unbiased walks may follow them too
  ctx->records_all_usable = ctx->V == 0 || (ctx->h_sum[3] & 0xFFFFFFFFull) == 0;
  return SKW_OK;
}

int skw_ctx_take_sampled_edges(skw_ctx* ctx, uint64_t* out) {
  if (!ctx) return SKW_ERR_ARG;
  DeviceGuard g(ctx->device);
  const int rc = err_check(ctx, "enqueued walks", true);  // synchronises the stream
  if (rc != SKW_OK) return rc;
  const uint64_t v = ctx->h_sum[1];
  if (out) *out = v;
  return SKW_OK;
}

int skw_probe_random_gather(skw_ctx* ctx, uint64_t footprint_bytes, uint32_t iters, double* gaccesses_per_s) {
  if (!ctx || !gaccesses_per_s) return SKW_ERR_ARG;
  if (footprint_bytes < (1ull << 20) || iters == 0)
    return fail(ctx, SKW_ERR_ARG, "skw_probe_random_gather: need a footprint of at least 1 MiB and iters > 0");
  DeviceGuard g(ctx->device);
  const u64 nrec = footprint_bytes / sizeof(WalkRecord);
  WalkRecord* buf = nullptr;
  SKW_CUDA(ctx, dev_malloc(ctx, &buf, nrec * sizeof(WalkRecord)));
  cudaStream_t st = ctx->stream;
  cudaError_t e = cudaMemsetAsync(buf, 1, nrec * sizeof(WalkRecord), st);
  const int grid = ctx->sm_count * 8;
  unsigned long long* sink = reinterpret_cast<unsigned long long*>(ctx->d_sum) + 1;
  float ms = 0;
  if (e == cudaSuccess) {
    probe_gather_kernel<<<grid, 256, 0, st>>>(buf, nrec, 8, sink);  // warm-up
    cudaEventRecord(ctx->ev0, st);
    probe_gather_kernel<<<grid, 256, 0, st>>>(buf, nrec, iters, sink);
    cudaEventRecord(ctx->ev1, st);
    ctx->launches += 2;
    e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  }
  dev_free(buf);
  if (e != cudaSuccess) return fail_cuda(ctx, e, "skw_probe_random_gather", __FILE__, __LINE__);
  *gaccesses_per_s = (double)grid * 256.0 * iters / (ms * 1e-3) / 1e9;
  return SKW_OK;
}

int skw_walk_records_free(skw_ctx* ctx) {
  if (!ctx) return SKW_ERR_ARG;
  DeviceGuard g(ctx->device);
  SKW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  dev_free(ctx->records);
  dev_free(ctx->vinfo);
  dev_free(ctx->vbits);
  dev_give_back(ctx->device);
  ctx->records = nullptr;
  ctx->vinfo = nullptr;
  ctx->vbits = nullptr;
  ctx->records_ready = false;
  return SKW_OK;
}

// Argument and state checks shared by the walk entry points.
static int walk_check(skw_ctx* ctx, const skw_walk_params* prm) {
  if (prm->hop_num < 1) return fail(ctx, SKW_ERR_ARG, "skw_walk: hop_num must be >= 1");
  if (prm->app > SKW_APP_NODE2VEC) return fail(ctx, SKW_ERR_ARG, "skw_walk: unknown app %u", prm->app);
  if (prm->mode > SKW_MODE_ONLINE) return fail(ctx, SKW_ERR_ARG, "skw_walk: unknown mode %u", prm->mode);
  if (prm->app == SKW_APP_PPR && !(prm->tp >= 0.0f && prm->tp <= 1.0f))
    return fail(ctx, SKW_ERR_ARG, "skw_walk: tp must be in [0,1]");
  if (prm->app == SKW_APP_NODE2VEC && !(prm->p > 0.0f && prm->q > 0.0f))
    return fail(ctx, SKW_ERR_ARG, "skw_walk: p and q must be positive");
  if (!ctx->xadj) return fail(ctx, SKW_ERR_STATE, "skw_walk: no graph resident");
  const bool unbiased = (prm->flags & SKW_WALK_UNBIASED) != 0;
  const bool online = prm->mode == SKW_MODE_ONLINE && !unbiased;
  if (!online && !unbiased && !ctx->table_ready)
    return fail(ctx, SKW_ERR_STATE, "skw_walk: offline mode needs skw_alias_build_offline or skw_alias_import first");
  if (online && !ctx->adjwgt) return fail(ctx, SKW_ERR_STATE, "skw_walk: online mode needs the edge weights");
  return SKW_OK;
}

// Whether an online batch is better served by building the tables of the whole graph (into memory of its own, for this
// call) than by computing its slots one by one.  A slot computed from the weights costs 2.7 ns of a full GPU and 7.5 us
// of a walker's time, and the first visit of a list 25 ns a weight of it (a batch that makes enough steps to meet the
// longest list waits for that); a table costs 10 ps an edge of the graph and some 60 us to launch, and a step over it 0.15 ns or
// 1.2 us.  40,000 x 80 node2vec on 204 M edges: 8.7 ms computed, 2.6 ms with tables; 256 x 80 on 4 M edges: 0.61
// against 0.2 ms; 256 x 5 on 117 M edges is 0.04 ms computed.  The figures are those of a B200; where the line
// lies exactly matters little, since near it both ways take the same time.
static bool tables_pay(const skw_ctx* ctx, const skw_walk_params* prm, uint64_t n) {
  double longest = prm->hop_num - 1.0, steps = longest;
  if (prm->app == SKW_APP_PPR && prm->tp > 0.0f) {
    longest = std::min(longest, (log((double)n) + 1.0) / prm->tp);
    steps = std::min(steps, 1.0 / prm->tp);
  }
  steps *= (double)n;
  const double hub = steps * ctx->max_degree >= (double)ctx->E ? 25e-9 * ctx->max_degree : 0.0;
  const double computed = std::max(7.5e-6 * longest + hub, 2.7e-9 * steps);
  const double tables = 60e-6 + 10e-12 * (double)ctx->E + std::max(1.2e-6 * longest, 0.15e-9 * steps);
  return tables < computed;
}

// Memory for such tables: 8 bytes an edge, and what the builders need.  False when there is none to be had.
static bool online_table_memory(skw_ctx* ctx) {
  if ((ctx->online_slots || dev_malloc(ctx, &ctx->online_slots, sizeof(Slot) * (ctx->E ? ctx->E : 1)) == cudaSuccess) &&
      (ctx->online_valid || dev_malloc(ctx, &ctx->online_valid, ctx->V ? ctx->V : 1) == cudaSuccess) &&
      reserve_builders(ctx, ctx->V) == SKW_OK)
    return true;
  cudaGetLastError();
  return false;
}

// Tables of the whole graph for one online call; slots is null if it does without.
struct OnlineTables {
  skw_ctx* ctx;
  const Slot* slots = nullptr;
  explicit OnlineTables(skw_ctx* c) : ctx(c) {}
  ~OnlineTables() { ctx->online_in_use = false; }
};

// Queue such tables for the n walkers of a call, where they pay.
static int online_tables(const skw_walk_params* prm, uint64_t n, OnlineTables& t) {
  skw_ctx* ctx = t.ctx;
  if (prm->mode != SKW_MODE_ONLINE || !n ||
      (prm->flags & (SKW_WALK_UNBIASED | SKW_WALK_CACHE_TABLES | SKW_WALK_BUILD_TABLES | SKW_WALK_DIRECT_SLOTS)))
    return SKW_OK;
  // A graph would keep the addresses of this memory, which can be given up or grow once the call is over.
  if (!tables_pay(ctx, prm, n) || capturing(ctx)) return SKW_OK;
  ctx->online_in_use = true;
  if (!online_table_memory(ctx)) {
    ctx->online_in_use = false;  // computing slots takes memory as well
    return SKW_OK;
  }
  const int rc = enqueue_tables(ctx, 0, ctx->V, ctx->online_slots, ctx->online_valid);
  if (rc == SKW_OK) t.slots = ctx->online_slots;
  return rc;
}

// Whether a call builds the tables of its walkers' vertices at every step.
static bool builds_frontiers(const skw_walk_params* prm) {
  return prm->mode == SKW_MODE_ONLINE && !(prm->flags & SKW_WALK_UNBIASED) &&
         (prm->flags & (SKW_WALK_CACHE_TABLES | SKW_WALK_BUILD_TABLES)) != 0;
}

// Walk records serve unbiased walks as well (the record of column c names the c-th neighbour with its offset and degree: one
// access per step instead of two), as long as every vertex with out-edges has a usable table, i.e. the degrees in the records
// are the graph's own.
static bool follows_records(const skw_ctx* ctx, const skw_walk_params* prm) {
  const bool unbiased = (prm->flags & SKW_WALK_UNBIASED) != 0;
  return (prm->mode != SKW_MODE_ONLINE || unbiased) && ctx->records_ready && prm->app != SKW_APP_NODE2VEC &&
         (!unbiased || ctx->records_all_usable);
}
// PPR over the records by chunks.  The kernel hands a lane its next walker cheaply; a batch with a lane for every walker,
// resident at once, does not need that (4,096 walkers: 29 -> 26 us, 100,000: 40 -> 38, equal at 200,000, 81 -> 89 at
// 400,000).  It stages lengths as 16-bit values and has no grid-stride loop.
static u64 ppr_chunk_ctas(u64 n) { return (n + 8 * kChunk - 1) / (8 * kChunk); }
static bool ppr_by_chunks(const skw_ctx* ctx, const skw_walk_params* prm, u64 n) {
  return follows_records(ctx, prm) && prm->app == SKW_APP_PPR && prm->hop_num <= 65535 && ppr_chunk_ctas(n) <= 0x7FFFFFFFull &&
         n > 700ull * ctx->sm_count;
}

// Queue the kernels of one batch of walkers on the context's stream; sampled edges are added to *sum.
// No reset, no readback, no synchronisation (the online paths allocate on first use).  whole_table: the
// slots that online_tables gave for the call.  d_heads: where ppr_by_chunks may leave the first cells of the rows instead.
// home: the rows are written_home's.
static int walk_launch(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* d_starts, uint64_t n,
                       uint32_t* d_paths, uint32_t* d_lengths, unsigned long long* sum, const Slot* whole_table,
                       uint32_t* d_heads = nullptr, bool home = false) {
  const bool unbiased = (prm->flags & SKW_WALK_UNBIASED) != 0;
  const bool online = prm->mode == SKW_MODE_ONLINE && !unbiased;
  int rc;
  // Online walks make one launch over tables of the whole graph or one that computes every slot it draws, whichever
  // pays; on request they build the tables of the frontier at every step (same walks).
  const bool build_tables = builds_frontiers(prm);
  if (build_tables) {
    drop_records(ctx);  // online builds overwrite table slots
    if ((rc = alloc_table(ctx, TableUse::kFrontier)) != SKW_OK) return rc;
  }
  if (!n) return SKW_OK;
  WalkArgs a;
  a.xadj = ctx->xadj;
  a.adjncy = ctx->adjncy;
  a.slots = ctx->slots;
  a.starts = d_starts;
  a.paths = d_paths;
  a.lengths = d_lengths;
  a.sum = sum;
  a.err = ctx->launch_err;
  a.n = n;
  a.seed = prm->seed;
  a.walker_base = prm->walker_base;
  a.walker_stride = prm->walker_stride ? prm->walker_stride : 1;
  a.V = ctx->V;
  a.hop_num = prm->hop_num;
  a.unbiased = unbiased ? 1u : 0u;
  a.tp = prm->tp;
  a.inv_p = prm->app == SKW_APP_NODE2VEC ? 1.0f / prm->p : 1.0f;
  a.inv_q = prm->app == SKW_APP_NODE2VEC ? 1.0f / prm->q : 1.0f;
  a.fmax = fmaxf(1.0f, fmaxf(a.inv_p, a.inv_q));
  cudaStream_t st = ctx->stream;
  if (whole_table) a.slots = whole_table;
  if (follows_records(ctx, prm)) {
    RecordWalkArgs ra;
    ra.unbiased = unbiased ? 1u : 0u;
    ra.rec = static_cast<const WalkRecord*>(ctx->records);
    ra.vinfo = static_cast<const uint2*>(ctx->vinfo);
    ra.vbits = static_cast<const u32*>(ctx->vbits);
    ra.starts = d_starts;
    ra.paths = d_paths;
    ra.heads = d_heads;
    ra.lengths = d_lengths;
    ra.sum = a.sum;
    ra.err = a.err;
    ra.n = n;
    ra.seed = a.seed;
    ra.walker_base = a.walker_base;
    ra.walker_stride = a.walker_stride;
    ra.V = a.V;
    ra.hop_num = a.hop_num;
    ra.tp = a.tp;
    const WalkGrid g = walk_grid(ctx, prm->app, n, 17, 8);
    if (ppr_by_chunks(ctx, prm, n)) {
      walk_records_ppr_kernel<8, kChunk, kStage><<<(unsigned)ppr_chunk_ctas(n), 256, 0, st>>>(ra);
    } else if (prm->app == SKW_APP_PPR) walk_records_walk_kernel<SKW_APP_PPR><<<g.ctas, kWalkCta, 0, st>>>(ra, g.lanes);
    else walk_records_walk_kernel<SKW_APP_DEEPWALK><<<g.ctas, kWalkCta, 0, st>>>(ra, g.lanes);
    SKW_LAUNCHED(ctx);
  } else if (!online || whole_table) {
    const u64 read = ctx->E * (unbiased ? 4u : 12u);  // lists, and slots if they are drawn from
    const WalkGrid g = walk_grid(ctx, prm->app, n, prm->app == SKW_APP_DEEPWALK && read <= (8u << 20) ? 17 : 34, 1);
    const bool ahead = walk_ahead(ctx, prm->app, n, prm->hop_num, unbiased);
    const size_t rings = home ? sizeof(u32) * (kWalkCta / 32) * g.lanes * (kLineRing + 1) : 0;
    switch (prm->app) {
      case SKW_APP_DEEPWALK:
        if (home && ahead) walk_home_kernel<SKW_APP_DEEPWALK, true><<<g.ctas, kWalkCta, rings, st>>>(a, g.lanes);
        else if (home) walk_home_kernel<SKW_APP_DEEPWALK, false><<<g.ctas, kWalkCta, rings, st>>>(a, g.lanes);
        else if (ahead) walk_offline_kernel<SKW_APP_DEEPWALK, true><<<g.ctas, kWalkCta, 0, st>>>(a, g.lanes);
        else walk_offline_kernel<SKW_APP_DEEPWALK, false><<<g.ctas, kWalkCta, 0, st>>>(a, g.lanes);
        break;
      case SKW_APP_PPR:
        if (home && ahead) walk_home_kernel<SKW_APP_PPR, true><<<g.ctas, kWalkCta, rings, st>>>(a, g.lanes);
        else if (home) walk_home_kernel<SKW_APP_PPR, false><<<g.ctas, kWalkCta, rings, st>>>(a, g.lanes);
        else if (ahead) walk_offline_kernel<SKW_APP_PPR, true><<<g.ctas, kWalkCta, 0, st>>>(a, g.lanes);
        else walk_offline_kernel<SKW_APP_PPR, false><<<g.ctas, kWalkCta, 0, st>>>(a, g.lanes);
        break;
      default: {
        const unsigned ctas = (unsigned)std::min<u64>((n + kN2vCta - 1) / kN2vCta, 0x7FFFFFFFull);
        switch (n2v_way(ctx, prm, n, unbiased)) {
          case N2vWay::kAccess: walk_n2v_kernel<<<ctas, kN2vCta, 0, st>>>(a); break;
          case N2vWay::kStep: walk_n2v_steps_kernel<false><<<ctas, kN2vCta, 0, st>>>(a); break;
          case N2vWay::kStepHalving: walk_n2v_steps_kernel<true><<<ctas, kN2vCta, 0, st>>>(a); break;
        }
        break;
      }
    }
    SKW_LAUNCHED(ctx);
  } else if (!build_tables) {
    if ((rc = launch_walk_online_direct(ctx, a, prm->app)) != SKW_OK) return rc;
  } else {
    const int grid = grid_for(ctx, n, 8);
    walk_online_init_kernel<<<grid, 256, 0, st>>>(a);
    SKW_LAUNCHED(ctx);
    for (uint32_t step = 0; step + 1 < prm->hop_num; ++step) {
      if ((rc = frontier_collect(ctx, d_paths, n, 1, prm->hop_num, step, d_lengths,
                                 step == 0 || !(prm->flags & SKW_WALK_CACHE_TABLES))) != SKW_OK) return rc;
      switch (prm->app) {
        case SKW_APP_DEEPWALK: walk_online_step_kernel<SKW_APP_DEEPWALK><<<grid, 256, 0, st>>>(a, step); break;
        case SKW_APP_PPR: walk_online_step_kernel<SKW_APP_PPR><<<grid, 256, 0, st>>>(a, step); break;
        default: walk_online_step_kernel<SKW_APP_NODE2VEC><<<grid, 256, 0, st>>>(a, step); break;
      }
      SKW_LAUNCHED(ctx);
    }
  }
  return SKW_OK;
}

// A synchronous walk over device buffers; with h_lengths the lengths, with h_paths the whole matrix comes home as well.
static int walk_and_wait(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* d_starts, uint64_t n, uint32_t* d_paths,
                         uint32_t* d_lengths, uint32_t* h_lengths, uint32_t* h_paths, float* ms,
                         uint64_t* sampled_edges, bool home = false) {
  cudaStream_t st = ctx->stream;
  int rc = err_reset(ctx);
  if (rc != SKW_OK) return rc;
  if (ms) SKW_CUDA(ctx, cudaEventRecord(ctx->ev0, st));
  OnlineTables tables(ctx);
  if ((rc = online_tables(prm, n, tables)) != SKW_OK) return rc;
  if ((rc = walk_launch(ctx, prm, d_starts, n, d_paths, d_lengths, reinterpret_cast<unsigned long long*>(ctx->d_sum),
                        tables.slots, nullptr, home)) != SKW_OK)
    return rc;
  if (ms) SKW_CUDA(ctx, cudaEventRecord(ctx->ev1, st));
  if (h_lengths && n) SKW_CUDA(ctx, cudaMemcpyAsync(h_lengths, d_lengths, sizeof(u32) * (size_t)n, cudaMemcpyDeviceToHost, st));
  if (h_paths && n)
    SKW_CUDA(ctx, cudaMemcpyAsync(h_paths, d_paths, sizeof(u32) * (size_t)n * prm->hop_num, cudaMemcpyDeviceToHost, st));
  if ((rc = err_check(ctx, "skw_walk")) != SKW_OK) return rc;
  if (ms) SKW_CUDA(ctx, cudaEventElapsedTime(ms, ctx->ev0, ctx->ev1));
  if (sampled_edges) *sampled_edges = *ctx->h_sum;
  return SKW_OK;
}

int skw_walk_device(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* d_starts, uint64_t n,
                    uint32_t* d_paths, uint32_t* d_lengths, float* ms, uint64_t* sampled_edges) {
  if (!ctx || !prm) return SKW_ERR_ARG;
  if (n && (!d_starts || !d_paths || !d_lengths))
    return fail(ctx, SKW_ERR_ARG, "skw_walk: null buffer");
  int rc = walk_check(ctx, prm);
  if (rc != SKW_OK) return rc;
  DeviceGuard g(ctx->device);
  // With both result pointers null the call only enqueues work: no reset, no readback, no
  // synchronisation.  Sampled edges then add up in a second counter and a device error stays
  // in a second record until skw_ctx_take_sampled_edges() looks at them.
  if (!ms && !sampled_edges) {
    QueuedErrors q(ctx);
    ctx->queued = true;
    OnlineTables tables(ctx);
    if ((rc = online_tables(prm, n, tables)) != SKW_OK) return rc;
    rc = walk_launch(ctx, prm, d_starts, n, d_paths, d_lengths, reinterpret_cast<unsigned long long*>(ctx->d_sum) + 1,
                     tables.slots);
    const int after = tables.slots || builds_frontiers(prm) ? builders_queued(ctx) : SKW_OK;
    return rc != SKW_OK ? rc : after;
  }
  return walk_and_wait(ctx, prm, d_starts, n, d_paths, d_lengths, nullptr, nullptr, ms, sampled_edges);
}

// Large batches into the caller's n x hop_num host matrix: the walks come home packed (contiguous
// copies, only cells that hold a vertex cross the bus) into pinned staging owned by the context, and
// host threads scatter them into the rows.  A kernel writing row prefixes straight into mapped host
// memory sends one small bus write per row (8 M PPR rows: 22 ms); a copy of the whole matrix moves
// every unused cell as well.  Cells past a walk's end keep what the caller had there.
static int walk_rows_by_scatter(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* h_starts, uint64_t n,
                                uint32_t* h_paths, uint32_t* h_lengths, float* ms, uint64_t* sampled_edges) {
  const uint64_t full = n * prm->hop_num;
  uint64_t want = full;
  if (prm->app == SKW_APP_PPR && prm->tp > 0.0f)
    want = std::min<uint64_t>(full, (uint64_t)((double)n * (1.0 / prm->tp + 2.0)) + 4096);
  uint64_t cells = 0;
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (ctx->h_pack_cells < want) {
      if (ctx->h_pack) cudaFreeHost(ctx->h_pack);
      ctx->h_pack = nullptr;
      ctx->h_pack_cells = 0;
      SKW_CUDA(ctx, cudaMallocHost(&ctx->h_pack, sizeof(uint32_t) * (size_t)want));
      ctx->h_pack_cells = want;
    }
    const int rc = skw_walk_packed(ctx, prm, h_starts, n, ctx->h_pack, ctx->h_pack_cells, h_lengths, &cells, ms,
                                   sampled_edges);
    if (rc == SKW_OK) break;
    if (rc != SKW_ERR_ARG || cells <= ctx->h_pack_cells || attempt == 1) return rc;
    want = std::min<uint64_t>(full, cells + (cells >> 3) + 4096);  // the staging was too small: once more
  }
  if (!ctx->host_pool) {
    unsigned hc = std::thread::hardware_concurrency();
    ctx->host_pool = new HostPool((int)std::min<unsigned>(hc ? hc : 1u, 32u));
  }
  HostPool* pool = static_cast<HostPool*>(ctx->host_pool);
  const int T = pool->size();
  std::vector<uint64_t> first(T + 1, 0);  // cells before each thread's block of walkers
  const uint32_t hop = prm->hop_num;
  pool->run([&](int t, int) {
    const uint64_t lo = n * t / T, hi = n * (t + 1) / T;
    uint64_t sum = 0;
    for (uint64_t w = lo; w < hi; ++w) sum += (uint64_t)std::min<uint32_t>(h_lengths[w] + 1u, hop);
    first[t + 1] = sum;
  });
  for (int t = 0; t < T; ++t) first[t + 1] += first[t];
  if (first[T] != cells)
    return fail(ctx, SKW_ERR_DEVICE, "skw_walk: packed result holds %llu cells, the lengths add up to %llu",
                (unsigned long long)cells, (unsigned long long)first[T]);
  const uint32_t* packed = ctx->h_pack;
  pool->run([&](int t, int) {
    const uint64_t lo = n * t / T, hi = n * (t + 1) / T;
    uint64_t o = first[t];
    // every row is a cache miss of its own (rows lie hop_num cells apart): ask for the lines a few rows
    // ahead, and copy short rows cell by cell (most PPR rows hold a handful of cells)
    constexpr uint64_t kAhead = 24;
    for (uint64_t w = lo; w < hi; ++w) {
      if (w + kAhead < hi) __builtin_prefetch(h_paths + (w + kAhead) * hop, 1, 0);
      const uint32_t c = std::min<uint32_t>(h_lengths[w] + 1u, hop);
      uint32_t* row = h_paths + w * hop;
      const uint32_t* src = packed + o;
      if (c <= 8) {
        for (uint32_t k = 0; k < c; ++k) row[k] = src[k];
      } else {
        memcpy(row, src, sizeof(uint32_t) * c);
      }
      o += c;
    }
  });
  return SKW_OK;
}

// `count` words of host memory as the GPU sees them, or null where it does not or where they are not at a word boundary.  All of
// them have to be in one pinned allocation or registration: parts of an array may be registered, with pages between them that
// the GPU must not touch.
static u32* seen_by_gpu(uint32_t* h, uint64_t count) {
  using Query = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
  static const Query query = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<Query>(f);
  }();
  cudaPointerAttributes at;
  if ((reinterpret_cast<uintptr_t>(h) & 3) != 0 || !query) return nullptr;
  if (cudaPointerGetAttributes(&at, h) != cudaSuccess || at.type != cudaMemoryTypeHost || !at.devicePointer) {
    cudaGetLastError();
    return nullptr;
  }
  const uint64_t d = reinterpret_cast<uint64_t>(at.devicePointer);
  CUdeviceptr start = 0;
  size_t size = 0;
  if (query(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, d) != CUDA_SUCCESS ||
      query(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, d) != CUDA_SUCCESS || d < start || d - start > size ||
      (size - (d - start)) / sizeof(u32) < count)
    return nullptr;
  return static_cast<u32*>(at.devicePointer);
}

// Whether walk_home_kernel takes a batch: as long as the walks, a chain of hop_num dependent steps whatever their number, hide
// most of the writes, which cross the bus at 36 GB/s where a copy behind the walks takes 52 (a sector a packet against whole
// lines).  Rows of a line or less are mostly ends of lines; what they gain is the copies and the clearing of the matrix that
// nobody has to queue, as long as every walker has a warp.  Calls, us, copied / written (R-MAT 16, 18, 20 and 22): 80 steps, 256
// walkers 163-197 / 135-152, 4,096 177-194 / 140-148, 16,000 274-291 / 202-209, 29,600 359-385 / 295-311, and with the same
// walks at every call 40,000 424-467 / 369-385, 80,000 642-809 / 681-722; 200 steps, 4,096 305-379 / 245-275, 16,000 539-605 /
// 356-410; 10 steps, 256 73-77 / 59-60, 5,000 84-88 / 72-74, 10,000 86-90 / 78-89, 20,000 97-102 / 106-115.  PPR of at most
// 100 steps, tp 0.15: 256 walkers 94-98 / 79-82, 4,096 151-165 / 108-112, 29,600 344-365 / 321-330.
// Beyond the end of the longest walk nothing hides the writes.  It is estimated from what ends a walk, the PPR draw and the
// edges into vertices without out-edges: the rows go home this way as long as the cells behind it are at most 2.5 MB, which is
// about what the copy's own launches cost, and at most 160 a row, which a warp writes one line after another.  Copied /
// written: PPR, tp 0.15, R-MAT 18, 4,096 x 201 185 / 150, 29,600 x 81 325 / 321, but 10,000 x 501 491 / 563, 29,600 x 201
// 579 / 626, 256 x 1,001 125 / 188; DeepWalk on a graph whose walks are over after a step 4,096 x 81 98 / 92, but
// 29,600 x 81 266 / 329, 4,096 x 501 223 / 230, 29,600 x 33 164 / 178; on R-MAT 18, where one edge of a hundred (directed)
// or none leads to such a vertex, 29,600 x 201 799 / 675 and 805 / 629, 4,096 x 1,001 1,194 / 943 and 1,316 / 1,089.
// Only where the whole matrix comes home whatever happens, as it does where rows are filled.  Where they are not, cells past
// a walk's end keep what the caller had there, and so do all of them when a walk meets a vertex that does not exist: rows are
// not written before the whole batch is known to be good.
static bool written_home(const skw_ctx* ctx, const skw_walk_params* prm, uint64_t n) {
  if (n == 0 || !(prm->flags & SKW_WALK_FILL_ROWS) || prm->app == SKW_APP_NODE2VEC) return false;
  const double into_ends = (double)ctx->dead_ends / skw_ctx::kEdgeSample;
  const double stop = prm->app == SKW_APP_PPR ? prm->tp + (1.0 - prm->tp) * into_ends : into_ends;  // a step's chance to be the last
  const double longest = stop <= 0.0 ? prm->hop_num : stop >= 1.0 ? 0.0 : log((double)n) / -log1p(-stop);
  const double behind = prm->hop_num - std::min<double>(prm->hop_num, longest);
  if (behind > 160.0 || behind * (double)n * sizeof(u32) > 2.5e6) return false;
  return n <= (prm->hop_num > kLineCells ? 200ull : 34ull) * ctx->sm_count &&
         prm->hop_num <= (1u << 24) &&  // the kernel counts up to a line past the row's end in 32 bits
         (prm->mode != SKW_MODE_ONLINE || (prm->flags & SKW_WALK_UNBIASED)) && !follows_records(ctx, prm);
}

int skw_walk(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* h_starts, uint64_t n,
             uint32_t* h_paths, uint32_t* h_lengths, float* ms, uint64_t* sampled_edges) {
  if (!ctx || !prm) return SKW_ERR_ARG;
  if (n && (!h_starts || !h_paths || !h_lengths)) return fail(ctx, SKW_ERR_ARG, "skw_walk: null buffer");
  if (prm->hop_num < 1) return fail(ctx, SKW_ERR_ARG, "skw_walk: hop_num must be >= 1");
  DeviceGuard g(ctx->device);
  int rc = walk_check(ctx, prm);
  if (rc != SKW_OK) return rc;
  if (n >= (1u << 18)) {
    if (prm->flags & SKW_WALK_FILL_ROWS) memset(h_paths, 0xFF, sizeof(uint32_t) * (size_t)n * prm->hop_num);
    return walk_rows_by_scatter(ctx, prm, h_starts, n, h_paths, h_lengths, ms, sampled_edges);
  }
  const size_t nb = sizeof(uint32_t) * (size_t)n;
  if ((rc = ensure_bytes(ctx, &ctx->stage[0], &ctx->stage_bytes[0], nb)) != SKW_OK) return rc;
  if (written_home(ctx, prm, n)) {
    u32* const rows = seen_by_gpu(h_paths, n * prm->hop_num);
    u32* const lengths = rows ? seen_by_gpu(h_lengths, n) : nullptr;
    if (lengths) {
      SKW_CUDA(ctx, cudaMemcpyAsync(ctx->stage[0], h_starts, nb, cudaMemcpyHostToDevice, ctx->stream));
      return walk_and_wait(ctx, prm, static_cast<uint32_t*>(ctx->stage[0]), n, rows, lengths, nullptr, nullptr, ms, sampled_edges,
                           true);
    }
  }
  if ((rc = ensure_bytes(ctx, &ctx->stage[1], &ctx->stage_bytes[1], nb * prm->hop_num)) != SKW_OK) return rc;
  if ((rc = ensure_bytes(ctx, &ctx->stage[2], &ctx->stage_bytes[2], nb)) != SKW_OK) return rc;
  if (n) SKW_CUDA(ctx, cudaMemcpyAsync(ctx->stage[0], h_starts, nb, cudaMemcpyHostToDevice, ctx->stream));
  const bool fill = (prm->flags & SKW_WALK_FILL_ROWS) != 0;
  if (n && fill) SKW_CUDA(ctx, cudaMemsetAsync(ctx->stage[1], 0xFF, nb * prm->hop_num, ctx->stream));
  uint64_t edges = 0;
  rc = walk_and_wait(ctx, prm, static_cast<uint32_t*>(ctx->stage[0]), n, static_cast<uint32_t*>(ctx->stage[1]),
                     static_cast<uint32_t*>(ctx->stage[2]), h_lengths, fill ? h_paths : nullptr, ms, &edges);
  if (rc != SKW_OK) return rc;
  if (sampled_edges) *sampled_edges = edges;
  if (n && !fill) {
    // Pinned host memory is addressable by the GPU: write only the cells each walk produced, unless that is all of
    // them (4096 rows of 81: one copy takes 31 us, the kernel 65).  Pageable memory gets the whole matrix (cells past a walk's
    // end then hold stale values).
    u32* const mapped = edges == n * (prm->hop_num - 1ull) ? nullptr : seen_by_gpu(h_paths, n * prm->hop_num);
    if (mapped) {
      copy_row_prefixes_kernel<<<ctx->sm_count * 8, 256, 0, ctx->stream>>>(
          static_cast<const u32*>(ctx->stage[1]), mapped, static_cast<const u32*>(ctx->stage[2]), n, prm->hop_num);
      SKW_LAUNCHED(ctx);
    } else {
      SKW_CUDA(ctx, cudaMemcpyAsync(h_paths, ctx->stage[1], nb * prm->hop_num, cudaMemcpyDeviceToHost, ctx->stream));
    }
    SKW_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return SKW_OK;
}

}  // extern "C"

// The packed host entry points: lengths come home as 32-bit words (h_lengths) or, for walks of at
// most 256 vertices, as bytes (h_lengths8); exactly one of the two is given.  use_heads: where that pays and there is memory.
static int walk_packed_impl(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* h_starts, uint64_t n,
                            uint32_t* h_packed, uint64_t capacity_cells, uint32_t* h_lengths,
                            uint8_t* h_lengths8, uint64_t* cells, float* ms, uint64_t* sampled_edges, bool use_heads = true) {
  if (!ctx || !prm) return SKW_ERR_ARG;
  if (!cells) return fail(ctx, SKW_ERR_ARG, "skw_walk_packed: cells must not be null");
  *cells = 0;
  if (ms) *ms = 0;
  if (sampled_edges) *sampled_edges = 0;
  if (n && (!h_starts || (!h_lengths && !h_lengths8))) return fail(ctx, SKW_ERR_ARG, "skw_walk_packed: null buffer");
  int rc = walk_check(ctx, prm);
  if (rc != SKW_OK) return rc;
  if (h_lengths8 && prm->hop_num > 256)
    return fail(ctx, SKW_ERR_ARG, "skw_walk_packed_u8: a length of up to %u does not fit a byte", prm->hop_num - 1);
  if (!n) return SKW_OK;
  DeviceGuard g(ctx->device);
  cudaStream_t st = ctx->stream, side = ctx->side_stream;
  // Large batches run as up to eight slices.  Everything a slice needs on the device (walk, prefix sum
  // of its row sizes, packing) is queued for ALL slices before the host waits for anything; the side
  // stream brings each slice's cell count, lengths and packed rows home as soon as they exist, while
  // the context's stream is already walking the next slice (the bus carries both directions at once).
  // Walker ids, hence walks, do not depend on the slicing.
  const uint64_t kSliceMin = 1u << 19;
  const uint32_t slices = n >= 8 * kSliceMin ? 8 : (n >= 4 * kSliceMin ? 4 : (n >= 2 * kSliceMin ? 3 : 1));
  static_assert(skw_ctx::kPackSlices >= 8 && skw_ctx::kStages >= 4 + 8, "one event set and one packing buffer per slice");
  // Slice sizes in the ratio 1 : 2 : 4 : 4 ... (three: 1 : 2 : 2): the first results are on the bus early (the call is
  // as long as the time to the first packed slice plus the copy of everything), the later slices are
  // large enough to walk efficiently.  2 M PPR walks: 926 us in two slices of 1 : 2, 880 in these three, 893 in four;
  // in two / three on R-MAT 20, 1.05, 1.3, 1.6 and 2 M walkers: PPR of 30 steps, tp 0.03, 1247 / 1178, 1506 / 1428, 1797 / 1777 and
  // 2257 / 2144, DeepWalk of ten steps 841 / 773, 916 / 912, 1098 / 1067 and 1414 / 1341.
  uint64_t base_of[skw_ctx::kPackSlices + 1] = {};
  uint64_t per = n;  // the largest slice
  if (slices > 1) {
    const uint64_t last = slices == 3 ? 2 : 4, parts = 3 + last * (slices - 2);
    const uint64_t unit = ((n + parts - 1) / parts + 1023) & ~1023ull;
    per = last * unit;
    for (uint32_t c = 0; c <= slices; ++c) {
      const uint64_t b = c == 0 ? 0 : (c == 1 ? unit : (3 + last * (c - 2)) * unit);
      base_of[c] = std::min<uint64_t>(b, n);
    }
  } else {
    base_of[1] = n;
  }
  const uint64_t stride = prm->walker_stride ? prm->walker_stride : 1;
  const size_t offs_bytes = (sizeof(u64) * (size_t)per + 255) & ~(size_t)255;
  size_t tmp_bytes = 0;
  {
    cub::TransformInputIterator<u64, CellsOfRow, const u32*> probe(static_cast<const u32*>(nullptr), CellsOfRow());
    SKW_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, probe, (u64*)nullptr, (long long)per, st));
  }
  if ((rc = ensure_bytes(ctx, &ctx->stage[0], &ctx->stage_bytes[0], sizeof(u32) * (size_t)n)) != SKW_OK) return rc;
  if ((rc = ensure_bytes(ctx, &ctx->stage[1], &ctx->stage_bytes[1], sizeof(u32) * (size_t)n * prm->hop_num)) != SKW_OK)
    return rc;
  if ((rc = ensure_bytes(ctx, &ctx->stage[2], &ctx->stage_bytes[2], sizeof(u32) * (size_t)n)) != SKW_OK) return rc;
  if ((rc = ensure_bytes(ctx, &ctx->stage[3], &ctx->stage_bytes[3], offs_bytes + tmp_bytes)) != SKW_OK) return rc;
  constexpr int kLen8Stage = 4 + skw_ctx::kPackSlices;
  constexpr int kHeadStage = skw_ctx::kHeadStage;
  static_assert(kHeadStage > kLen8Stage, "two more staging buffers for byte lengths and heads of rows");
  if (h_lengths8 && (rc = ensure_bytes(ctx, &ctx->stage[kLen8Stage], &ctx->stage_bytes[kLen8Stage], (size_t)n)) != SKW_OK)
    return rc;
  uint8_t* d_len8 = h_lengths8 ? static_cast<uint8_t*>(ctx->stage[kLen8Stage]) : nullptr;
  u32* d_starts = static_cast<u32*>(ctx->stage[0]);
  u32* d_rows = static_cast<u32*>(ctx->stage[1]);
  u32* d_len = static_cast<u32*>(ctx->stage[2]);
  u64* d_offs = static_cast<u64*>(ctx->stage[3]);
  // Packing buffers, one per slice.  The size of a result changes from call to call (another seed,
  // other lengths), so a buffer that exists is kept as it is and only a result that outgrows it makes
  // it grow (by an eighth more than needed): steady-state calls do not allocate.  First guess: every
  // walk at full length, or the expected PPR length with room to spare.
  uint64_t cap[skw_ctx::kPackSlices] = {}, nc_of[skw_ctx::kPackSlices] = {};
  for (uint32_t c = 0; c < slices; ++c) {
    const uint64_t base = base_of[c];
    if (base >= n) break;
    const uint64_t nc = base_of[c + 1] - base;
    nc_of[c] = nc;
    const uint64_t full = nc * prm->hop_num;
    uint64_t guess = full;
    if (prm->app == SKW_APP_PPR && prm->tp > 0.0f)
      guess = std::min<uint64_t>(full, (uint64_t)((double)nc * (1.0 / prm->tp + 2.0)) + 4096);
    if (ctx->stage[4 + c] && ctx->stage_bytes[4 + c] >= sizeof(u32) * 1024) guess = ctx->stage_bytes[4 + c] / sizeof(u32);
    if ((rc = ensure_bytes(ctx, &ctx->stage[4 + c], &ctx->stage_bytes[4 + c], sizeof(u32) * (size_t)guess)) != SKW_OK) return rc;
    cap[c] = std::min<uint64_t>(ctx->stage_bytes[4 + c] / sizeof(u32), full);
  }
  // PPR walks mostly end within the first cells of their rows.  Written to the rows, 404 bytes apart for 100 steps, these are
  // isolated sectors, a third of the walk's time, and read back as such; side by side both are streams.
  // Without memory for them the rows will do, so they come behind everything that the call cannot do without.
  const bool heads = use_heads && ppr_by_chunks(ctx, prm, n) &&
                     ensure_bytes(ctx, &ctx->stage[kHeadStage], &ctx->stage_bytes[kHeadStage],
                                  sizeof(u32) * kStage * (size_t)n) == SKW_OK;
  struct InUse {
    bool& flag;
    InUse(bool& f, bool used) : flag(f) { flag = used; }
    ~InUse() { flag = false; }
  } heads_in_use(ctx->heads_in_use, heads);
  bool outgrown = false;  // a packed slice for which there is no memory
  if ((rc = err_reset(ctx)) != SKW_OK) return rc;
  unsigned long long* scratch_sum = reinterpret_cast<unsigned long long*>(ctx->d_sum) + 2;
  auto heads_of = [&](uint32_t c) -> u32* {
    return heads && ppr_by_chunks(ctx, prm, nc_of[c]) ? static_cast<u32*>(ctx->stage[kHeadStage]) + base_of[c] * kStage : nullptr;
  };
  auto scan_and_pack = [&](uint32_t c) -> int {
    const uint64_t base = base_of[c], nc = nc_of[c];
    cub::TransformInputIterator<u64, CellsOfRow, const u32*> row_cells(d_len + base, CellsOfRow());
    size_t tb = tmp_bytes;
    SKW_CUDA(ctx, cub::DeviceScan::ExclusiveSum(reinterpret_cast<char*>(d_offs) + offs_bytes, tb, row_cells, d_offs,
                                                (long long)nc, st));
    SKW_LAUNCHED(ctx);
    // Packed on the device, then one contiguous copy per slice: measured on B200 with 8 M PPR walks,
    // half the time of a pack kernel that writes the pinned host buffer itself (its 4-byte stores
    // per row do not merge into full-size bus writes).
    u32* packed = static_cast<u32*>(ctx->stage[4 + c]);
    uint8_t* len8 = d_len8 ? d_len8 + base : nullptr;
    const u32* rows = d_rows + base * prm->hop_num;
    if (const u32* first = heads_of(c))
      pack_heads_kernel<<<grid_for(ctx, nc, 8), 256, 0, st>>>(rows, first, packed, d_len + base, d_offs, nc, prm->hop_num, cap[c],
                                                             ctx->h_tot + c, len8);
    else
      pack_rows_kernel<<<grid_for(ctx, nc * 8, 8), 256, 0, st>>>(rows, packed, d_len + base, d_offs, nc, prm->hop_num, cap[c],
                                                                ctx->h_tot + c, len8);
    SKW_LAUNCHED(ctx);
    SKW_CUDA(ctx, cudaEventRecord(ctx->pk_ready[c], st));
    SKW_CUDA(ctx, cudaStreamWaitEvent(side, ctx->pk_ready[c], 0));
    return SKW_OK;
  };
  // Times are taken on a stream of their own: a stream waits up to 40 us for its own timing event while copies are under way
  // (2 M PPR walks: 883 -> 869 us).
  auto take_time = [&](cudaEvent_t when) -> int {
    cudaStream_t clock = ctx->bstream[skw_ctx::kBuilderStreams - 1];
    SKW_CUDA(ctx, cudaEventRecord(ctx->bfork, st));
    SKW_CUDA(ctx, cudaStreamWaitEvent(clock, ctx->bfork, 0));
    SKW_CUDA(ctx, cudaEventRecord(when, clock));
    return SKW_OK;
  };
  OnlineTables tables(ctx);
  auto body = [&]() -> int {
    // the start vertices come in slice by slice on the side stream, ahead of everything else it will
    // carry: a walk waits for its own slice only, and no walk waits behind a copy of a later slice
    for (uint32_t c = 0; c < slices && nc_of[c]; ++c) {
      const uint64_t base = base_of[c], nc = nc_of[c];
      SKW_CUDA(ctx, cudaMemcpyAsync(d_starts + base, h_starts + base, sizeof(u32) * (size_t)nc, cudaMemcpyHostToDevice, side));
      SKW_CUDA(ctx, cudaEventRecord(ctx->pk_in[c], side));
    }
    for (uint32_t c = 0; c < slices && nc_of[c]; ++c) {
      const uint64_t base = base_of[c], nc = nc_of[c];
      SKW_CUDA(ctx, cudaStreamWaitEvent(st, ctx->pk_in[c], 0));
      skw_walk_params p = *prm;
      p.walker_base = prm->walker_base + base * stride;
      int r = take_time(ctx->pk_t0[c]);
      if (r == SKW_OK && c == 0) r = online_tables(prm, n, tables);  // for all slices
      if (r != SKW_OK) return r;
      r = walk_launch(ctx, &p, d_starts + base, nc, d_rows + base * prm->hop_num, d_len + base, scratch_sum, tables.slots,
                      heads_of(c));
      if (r != SKW_OK) return r;
      if ((r = take_time(ctx->pk_t1[c])) != SKW_OK || (r = scan_and_pack(c)) != SKW_OK) return r;
      if (h_lengths8)
        SKW_CUDA(ctx, cudaMemcpyAsync(h_lengths8 + base, d_len8 + base, (size_t)nc, cudaMemcpyDeviceToHost, side));
      else
        SKW_CUDA(ctx, cudaMemcpyAsync(h_lengths + base, d_len + base, sizeof(u32) * (size_t)nc, cudaMemcpyDeviceToHost, side));
    }
    ctx->online_in_use = false;  // every walk is queued, and freeing waits for the GPU
    // the host follows the device slice by slice: learn the size, start the copy
    uint64_t total_cells = 0;
    bool fits = h_packed != nullptr;
    float total_ms = 0;
    for (uint32_t c = 0; c < slices && nc_of[c]; ++c) {
      SKW_CUDA(ctx, cudaEventSynchronize(ctx->pk_ready[c]));
      uint64_t slice_cells = ctx->h_tot[c];
      if (fits && total_cells + slice_cells > capacity_cells) fits = false;  // keep going: the caller gets the size
      if (fits && slice_cells > cap[c]) {
        // this slice outgrew its packing buffer: grow it and pack once more (its rows and lengths are
        // still on the device).  Growing frees the old buffer, which waits for the device.
        const uint64_t roomy = std::min<uint64_t>(slice_cells + (slice_cells >> 3) + 4096, nc_of[c] * prm->hop_num);
        int r = ensure_bytes(ctx, &ctx->stage[4 + c], &ctx->stage_bytes[4 + c], sizeof(u32) * (size_t)roomy);
        if (r != SKW_OK) {
          outgrown = true;
          return r;
        }
        cap[c] = roomy;
        if ((r = scan_and_pack(c)) != SKW_OK) return r;
        SKW_CUDA(ctx, cudaEventSynchronize(ctx->pk_ready[c]));
        slice_cells = ctx->h_tot[c];
      }
      if (fits) {
        // on a stream of its own: the side stream already holds the (still waiting) count and length
        // copies of the later slices, and this copy must not queue up behind them
        SKW_CUDA(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->pk_ready[c], 0));
        SKW_CUDA(ctx, cudaMemcpyAsync(h_packed + total_cells, ctx->stage[4 + c], sizeof(u32) * (size_t)slice_cells,
                                      cudaMemcpyDeviceToHost, ctx->copy_stream));
      }
      total_cells += slice_cells;
      float t = 0;
      SKW_CUDA(ctx, cudaEventSynchronize(ctx->pk_t1[c]));  // (the walk is long over)
      SKW_CUDA(ctx, cudaEventElapsedTime(&t, ctx->pk_t0[c], ctx->pk_t1[c]));
      total_ms += t;
    }
    int r = err_check(ctx, "skw_walk_packed");  // synchronises the context's stream, while the last copies are under way
    SKW_CUDA(ctx, cudaStreamSynchronize(side));
    SKW_CUDA(ctx, cudaStreamSynchronize(ctx->copy_stream));
    if (r != SKW_OK) return r;
    *cells = total_cells;
    if (ms) *ms = total_ms;
    if (sampled_edges) *sampled_edges = total_cells - n;  // every walk holds its start plus one vertex per sampled edge
    if (!fits)
      return fail(ctx, SKW_ERR_ARG, "skw_walk_packed: the result needs %llu cells, the buffer holds %llu",
                  (unsigned long long)total_cells, (unsigned long long)(h_packed ? capacity_cells : 0));
    return SKW_OK;
  };
  rc = body();
  if (rc != SKW_OK && rc != SKW_ERR_ARG) {  // leave nothing in flight that still writes the caller's buffers
    const std::string why = ctx->err;
    cudaStreamSynchronize(side);
    cudaStreamSynchronize(ctx->copy_stream);
    cudaStreamSynchronize(st);
    ctx->err = why;
  }
  if (rc != SKW_OK && outgrown && heads) {  // the memory of the heads may be what is missing: once more without them
    ctx->heads_in_use = false;
    return walk_packed_impl(ctx, prm, h_starts, n, h_packed, capacity_cells, h_lengths, h_lengths8, cells, ms, sampled_edges, false);
  }
  return rc;
}

extern "C" {

int skw_walk_packed(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* h_starts, uint64_t n,
                    uint32_t* h_packed, uint64_t capacity_cells, uint32_t* h_lengths, uint64_t* cells,
                    float* ms, uint64_t* sampled_edges) {
  if (ctx && n && !h_lengths) return fail(ctx, SKW_ERR_ARG, "skw_walk_packed: null buffer");
  return walk_packed_impl(ctx, prm, h_starts, n, h_packed, capacity_cells, h_lengths, nullptr, cells, ms,
                          sampled_edges);
}

int skw_walk_packed_u8(skw_ctx* ctx, const skw_walk_params* prm, const uint32_t* h_starts, uint64_t n,
                       uint32_t* h_packed, uint64_t capacity_cells, uint8_t* h_lengths8, uint64_t* cells,
                       float* ms, uint64_t* sampled_edges) {
  if (ctx && n && !h_lengths8) return fail(ctx, SKW_ERR_ARG, "skw_walk_packed_u8: null buffer");
  return walk_packed_impl(ctx, prm, h_starts, n, h_packed, capacity_cells, nullptr, h_lengths8, cells, ms,
                          sampled_edges);
}

}  // extern "C"

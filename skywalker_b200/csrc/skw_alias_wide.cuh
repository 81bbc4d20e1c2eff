// Table of one weight list of 4097 to 16384 entries by a CTA of 512 or 1024 threads, in double precision and one tile in
// registers like the shorter lists (skw_alias_f64.cuh): 16 weights a thread, loaded and quantised once, two scans, one merge.
//
// What differs is that sums have up to 54 bits:
//   prefixes        D and X run from 0 to n * 2^40 and are kept less 2^53, where a double holds every integer.  A mass is exact
//                   below 2^53; a thread whose 16 weights have more (of more than 8192 weights, one with half of the total)
//                   goes the way of 64-bit integers.
//   running weight  up to 2^53 for 8192 weights, exact.  Beyond, it is counted from the multiple of 2^32 below its warp's
//                   start, so that one addition rounds it as the conversion of the 64-bit sum would be rounded.
//   list entry      8 bytes of key and 2 of position, in two arrays.
// The slots take the place of the keys as these are used up (merge_wide_step), so that two lists of 8192 weights fit an SM.
//
// Bound by the pipe of shared memory (70 % busy; put, bisection, merge and stores go to unrelated banks) and by barriers, with
// 158 warp instructions per 32 edges.  16.7 M edges in lists of 4097 / 6300 / 8192 weights: 238 / 218 / 200 us in tiles of
// eight weights a thread, each a pass for the largest weight and one for the total before it, and slots stored from the merge
// to where they belong; 174 / 153 / 153 us here.  9000 / 12000 / 16384 (one list an SM): 283 / 270 / 268 -> 216 / 191 / 192.
// Slots kept in the registers of the merging threads until all have read the lists: 194 / 179 / 159 (spills).  Clusters of two
// to eight CTAs of 512 threads for the lists beyond 8192, entries fetched out of one another's shared memory: 315 to 330 / 276
// to 290 / 262 to 269.
#pragma once
#include "skw_alias_f64.cuh"

namespace skw {

constexpr u32 kWideEpt = 16;
constexpr double kTwo53 = 2.0 * kTwo52;

// Cross-thread words of a CTA of NT threads.
template <int NT>
struct WideWords {
  static constexpr int NW = NT / 32;
  u64 q[NW], d[NW];
  u32 s[NW];
};

__device__ __forceinline__ u64 warp_scan_u64(u64 v, u32 lane, u64& total) {
  u64 inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u64 x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= (u32)o) inc += x;
  }
  total = __shfl_sync(0xFFFFFFFFu, inc, 31);
  return inc - v;
}

// Shared memory of a CTA: the staged weights, then the two lists.
template <u32 NT>
struct WideShared {
  static constexpr u32 kMost = NT * kWideEpt;
  union {
    struct {
      double key[kMost + 2];
      uint16_t pos[kMost + 2];
    };
    int stage[kMost + NT];  // an even number a thread is spread by one word a thread
  };
  WideWords<(int)NT> words;
  u64 first_q[NT / 32], total;  // running weight before each warp, and of the list
  u32 top[2][NT / 32];
};

// One list entry, stored if k < cnt: a small (c > 0) with the deficit before it at index is, a large with the excess up to
// and including it at index il; keys at shared address A, positions at P.
__device__ __forceinline__ void put_wide_entry(double c, u32 k, u32 cnt, u32 pos, u32 A, u32 P, double& D, double& X, u32& is,
                                               u32& il) {
  asm volatile(
      "{\n\t.reg .pred p, in;\n\t.reg .f64 key;\n\t.reg .b32 i, at;\n\t.reg .b16 h;\n\t"
      "setp.gt.f64 p, %4, 0d0000000000000000;\n\t"
      "setp.lt.u32 in, %5, %6;\n\t"
      "@!p sub.rn.f64 %1, %1, %4;\n\t"
      "selp.f64 key, %0, %1, p;\n\t"
      "selp.b32 i, %2, %3, p;\n\t"
      "@p add.rn.f64 %0, %0, %4;\n\t"
      "@p add.u32 %2, %2, 1;\n\t"
      "@!p sub.u32 %3, %3, 1;\n\t"
      "mad.lo.u32 at, i, 8, %8;\n\t"
      "@in st.shared.f64 [at], key;\n\t"
      "mad.lo.u32 at, i, 2, %9;\n\t"
      "cvt.u16.u32 h, %7;\n\t"
      "@in st.shared.u16 [at], h;\n\t}"
      : "+d"(D), "+d"(X), "+r"(is), "+r"(il)
      : "d"(c), "r"(k), "r"(cnt), "r"(pos), "r"(A), "r"(P)
      : "memory");
}

// One step of the merge (see merge_f64): smalls from the front of an array, the total deficit at end, larges from the array's
// back and an entry that is above all behind end.  sk, lk: keys of the heads, whose addresses are ps and pl; lp: position of
// the large one.  The slot of the entry that leaves is stored where the next head of its list was read: that of a small one
// entry further back, that of a large one entry further to the front.  Nobody needs that key any more, since all threads have
// read the heads that they begin with.  P: address of the positions less a quarter of that of the keys.
__device__ __forceinline__ void merge_wide_step(double& sk, double& lk, u32& lp, u32& ps, u32& pl, u32 end, u32 P) {
  asm volatile(
      "{\n\t.reg .pred take, more, whole;\n\t.reg .f64 was, key, mass;\n\t.reg .b32 at, of, old, alias, bits;\n\t.reg .f32 prob;\n\t"
      ".reg .b16 h;\n\t"
      "setp.ne.u32 more, %3, %5;\n\t"
      "setp.le.and.f64 take, %0, %1, more;\n\t"
      "selp.f64 was, %0, %1, take;\n\t"
      "mov.b32 old, %2;\n\t"
      "@take add.u32 %3, %3, 8;\n\t"
      "@!take sub.u32 %4, %4, 8;\n\t"
      "selp.b32 at, %3, %4, take;\n\t"
      "shr.u32 of, at, 2;\n\t"
      "add.u32 of, of, %6;\n\t"
      "ld.shared.f64 key, [at];\n\t"
      "@!take ld.shared.u16 h, [of];\n\t"
      "@!take cvt.u32.u16 %2, h;\n\t"
      "@take mov.f64 %0, key;\n\t"
      "@!take mov.f64 %1, key;\n\t"
      "sub.rn.f64 mass, was, %0;\n\t"
      "fma.rn.f64 mass, mass, 0d3D70000000000000, 0d3FF0000000000000;\n\t"  // in buckets (2^-40), exact
      "setp.ge.f64 whole, mass, 0d3FF0000000000000;\n\t"
      "selp.b32 alias, old, %2, whole;\n\t"
      "cvt.rn.f32.f64 prob, mass;\n\t"
      "mov.b32 bits, prob;\n\t"
      "st.shared.v2.b32 [at], {bits, alias};\n\t}"
      : "+d"(sk), "+d"(lk), "+r"(lp), "+r"(ps), "+r"(pl)
      : "r"(end), "r"(P)
      : "memory");
}

// g(Q) for Q = hi + rel; hi is the multiple of 2^32 below a warp's first running weight where sums may pass 2^53, else zero.
template <bool BIG>
struct WideMass {
  double hi, end, all, K;
  u32 h;
  __device__ __forceinline__ WideMass(u64 first, u64 W, u32 n) {
    h = BIG ? (u32)(first >> 32) : 0u;
    all = __ull2double_rn((u64)n << 40);
    K = __ddiv_rn(all, __ull2double_rn(W));
    hi = __dmul_rn(u32_to_double(h), 4294967296.0);
    end = __ull2double_rn(W - ((u64)h << 32));  // (exact where a thread may reach it)
  }
  __device__ __forceinline__ double rel(u64 q) const { return __ull2double_rn(q - ((u64)h << 32)); }
  // Up to 8192 weights Q * K never passes n * 2^40: W <= 2^53, so 1 - 1/W outweighs the rounding of K, and the product
  // rounds to n * 2^40 at most.
  __device__ __forceinline__ double operator()(double rel) const {
    const double g = trunc(__dmul_rn(BIG ? __dadd_rn(hi, rel) : rel, K));
    return rel == end || (BIG && g > all) ? all : g;
  }
};
// The quantised weight of bits b >= 0, finite, in a list whose largest weight has the bits top (at least 2^-87).
__device__ __forceinline__ double wide_quantised(int b, int top) {
  const u64 shift = (u64)(1062 - (top >> 23)) << 52;
  const double x = __longlong_as_double((long long)((u64)(u32)b * (1u << 29) + shift));
  return __dsub_rn(__dadd_rz(x, kTwo52), kTwo52);
}

// The lists that a CTA works through: places of the class's work list, handed out by its cursor.  Which one is next is asked
// for when a list is begun, told to all threads half-way, and its weights are on their way to L2 while the slots of this one
// are written.  Each step is called once a list, in this order, with a barrier before and behind tell().
struct WideItems {
  const u32* list;
  const u32* xadj;
  const float* wgt;
  u32* cursor;
  u32 count;
  u32* shared;         // a word of the CTA
  u32 v, off, end;     // the list
  u32 v1, off1, end1;  // the next one
  u32 asked;
  bool more;
  __device__ __forceinline__ void ask() {
    if (threadIdx.x == 0) asked = atomicAdd(cursor, 1u);
  }
  __device__ __forceinline__ void tell() const {
    if (threadIdx.x == 0) *shared = asked;
  }
  __device__ __forceinline__ void vertex() {
    const u32 it = *shared;
    more = it < count;
    v1 = more ? __ldg(list + it) : 0u;
  }
  __device__ __forceinline__ void offsets() {
    off1 = __ldg(xadj + v1);
    end1 = __ldg(xadj + v1 + 1);
  }
  __device__ __forceinline__ void weights() const {
    if (more && threadIdx.x * 32 < end1 - off1) asm volatile("prefetch.global.L2 [%0];" ::"l"(wgt + off1 + threadIdx.x * 32));
  }
  __device__ __forceinline__ void advance() {
    v = v1;
    off = off1;
    end = end1;
  }
};

template <u32 NT>
__device__ __forceinline__ void build_list_wide(u32 v, u32 off, u32 n, const float* __restrict__ w, Slot* __restrict__ slots,
                                                uint8_t* __restrict__ valid, WideShared<NT>* sh, u32* err, WideItems& items) {
  constexpr u32 NW = NT / 32, CH = 2;
  constexpr int EPT = (int)kWideEpt;
  constexpr bool kBig = NT * kWideEpt > 8192;
  const u32 t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const GroupCoop<32> wc;
  WideWords<(int)NT>& words = sh->words;
  const u32 ept = (n + NT - 1) / NT;
  const u32 p0 = min(t * ept, n), cnt = min(ept, n - p0);
  const u32 over = min((ept + CH - 1) / CH * CH, (u32)EPT) - cnt;
#define SKW_EACH(k)                                             \
  _Pragma("unroll") for (int b_ = 0; b_ < EPT; b_ += (int)CH) { \
    if ((u32)b_ >= ept) break;                                  \
    _Pragma("unroll") for (int k = b_; k < b_ + (int)CH; ++k)
#define SKW_EACH_END }
  int wb[EPT];
  {
    const u32 per = ept & 1 ? 0u : 0xFFFFFFFFu / ept + 1;  // i / ept as a multiplication (i < 2^14, ept <= 16)
#pragma unroll
    for (int k = 0; k < EPT; ++k) wb[k] = t + k * NT < n ? __float_as_int(__ldg(w + t + k * NT)) : 0;
    SKW_EACH(k) {
      const u32 i = t + k * NT;
      if (i < n) sh->stage[i + __umulhi(i, per)] = wb[k];
    }
    SKW_EACH_END
    __syncthreads();
    const int* mine = sh->stage + t * (ept | 1);
#pragma unroll
    for (int k = 0; k < EPT; ++k) wb[k] = (u32)k < cnt ? mine[k] : 0;
  }
  // the order of the bits of positive floats is the order of the values; what is negative (or minus zero) becomes zero
  int top = 0;
  SKW_EACH(k) {
    wb[k] = max(wb[k], 0);
    top = max(top, wb[k]);
  }
  SKW_EACH_END
  auto largest = [&](int use) {
    top = wc.template max<0>(top);
    if (lane == 0) sh->top[use][warp] = (u32)top;
    __syncthreads();
    top = wc.template max<0>(lane < NW ? (int)sh->top[use][lane] : 0);
  };
  largest(0);
  if (top >= 0x7F800000) {  // infinities and NaNs count as zero
    top = 0;
    SKW_EACH(k) {
      if (wb[k] >= 0x7F800000) wb[k] = 0;
      top = max(top, wb[k]);
    }
    SKW_EACH_END
    largest(1);
  }
  if (top == 0) {
    items.tell();
    for (u32 p = t; p < n; p += NT) slots[(u64)off + p] = Slot{-1.0f, p};
    if (t == 0) valid[v] = 0;
    __syncthreads();
    items.vertex();
    items.offsets();
    return;
  }
  // lists whose largest weight is below 2^-87 are scaled up (exactly), so that zeros and denormals quantise to 0
  const bool faint = top < (40 << 23);
  if (faint) {
    SKW_EACH(k) { wb[k] = __float_as_int(__int_as_float(wb[k]) * 18446744073709551616.0f); }
    SKW_EACH_END
    top = __float_as_int(__int_as_float(top) * 18446744073709551616.0f);
  }
  double c[EPT];
  double Q = 0.0, all;
  SKW_EACH(k) {
    c[k] = wide_quantised(wb[k], top);
    Q = __dadd_rn(Q, c[k]);
  }
  SKW_EACH_END
  wc.scan(Q, all);
  if (lane == 0) words.q[warp] = (u64)all;
  __syncthreads();
  u64 W, wq = warp_scan_u64(lane < NW ? words.q[lane] : 0, lane, W);
  wq = __shfl_sync(0xFFFFFFFFu, wq, warp);  // before this warp
  if (kBig) {
    if (lane == 0) sh->first_q[warp] = wq;
    if (t == 0) sh->total = W;
  }
  const u64 q0 = wq + (u64)Q;  // before this thread
  double g0, D = 0.0;
  u32 s = 0;
  bool giant;
  {
    const WideMass<kBig> mass(wq, W, n);
    double rel = __dadd_rn(Q, mass.rel(wq));
    g0 = mass(rel);
    double g = g0;
    SKW_EACH(k) {
      rel = __dadd_rn(rel, c[k]);
      const double gn = mass(rel);
      c[k] = __dsub_rn(kBucket, __dsub_rn(gn, g));  // what a small lacks, minus what a large has too much
      g = gn;
      count_small(c[k], D, s);
    }
    SKW_EACH_END
    giant = kBig && __dsub_rn(g, g0) >= kTwo53;
  }
  D = __dsub_rn(D, __dmul_rn((double)over, kBucket));
  s -= over;
  u32 all_s;
  wc.scan(D, s, all, all_s);
  if (lane == 0) {
    words.d[warp] = (u64)all;
    words.s[warp] = all_s;
  }
  __syncthreads();
  u64 tD, wd = warp_scan_u64(lane < NW ? words.d[lane] : 0, lane, tD);
  u32 S;
  {
    const u32 mine = lane < NW ? words.s[lane] : 0u;
    u32 inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= (u32)o) inc += y;
    }
    S = __shfl_sync(0xFFFFFFFFu, inc, 31);
    s += __shfl_sync(0xFFFFFFFFu, inc - mine, warp);
  }
  items.tell();
  constexpr u64 kMid = (u64)1 << 53;
  const u64 before = __shfl_sync(0xFFFFFFFFu, wd, warp) + (u64)D - kMid;  // deficit before this thread
  const u64 net = (u64)g0 - ((u64)p0 << 40);                               // excess minus deficit there
  const u32 A = (u32)__cvta_generic_to_shared(sh->key), P = (u32)__cvta_generic_to_shared(sh->pos);
  u32 is = s, il = n + 1 - (p0 - s);
  if (!giant) {
    D = __ll2double_rn((long long)before);
    double X = __ll2double_rn((long long)(before + net));
    SKW_EACH(k) { put_wide_entry(c[k], k, cnt, p0 + k, A, P, D, X, is, il); }
    SKW_EACH_END
  } else if constexpr (kBig) {
    // once more from the weights, with little kept for it
    const WideMass<kBig> mass(sh->first_q[warp], sh->total, n);
    u64 d = before, x = before + net, gi = (u64)g0;
    double rel = mass.rel(q0);
#pragma unroll 1
    for (u32 k = 0; k < cnt; ++k) {
      int b = max(__float_as_int(__ldg(w + p0 + k)), 0);
      if (b >= 0x7F800000) b = 0;
      if (faint) b = __float_as_int(__int_as_float(b) * 18446744073709551616.0f);
      rel = __dadd_rn(rel, wide_quantised(b, top));
      const u64 gn = (u64)mass(rel), m = gn - gi;
      gi = gn;
      const bool small = m < (1ull << 40);
      if (!small) x += m - (1ull << 40);
      const u32 i = small ? is : il;
      sh->key[i] = __ll2double_rn((long long)(small ? d : x));
      sh->pos[i] = (uint16_t)(p0 + k);
      if (small) d += (1ull << 40) - m;
      is += small ? 1u : 0u;
      il -= small ? 0u : 1u;
    }
  }
#undef SKW_EACH
#undef SKW_EACH_END
  if (t == 0) {
    sh->key[S] = __ll2double_rn((long long)(tD - kMid));
    sh->key[S + 1] = kTwo53 * kTwo53;
    sh->pos[S + 1] = 0;
  }
  __syncthreads();
  items.vertex();
  if (S >= n) {  // mass conservation guarantees a large
    if (t == 0) {
      dev_fail(err, DEV_ERR_INTERNAL, v, S, 7);
      valid[v] = 1;
    }
    for (u32 p = t; p < n; p += NT) slots[(u64)off + p] = Slot{1.0f, p};
    items.offsets();
    return;
  }
  items.offsets();
  // the merge, each thread an equal share
  const u32 L = n - S;
  is = p0 > L ? p0 - L : 0;
  {
    u32 up = min(p0, S);
    while (is < up) {
      const u32 mid = (is + up) >> 1;
      const bool first = sh->key[mid] <= sh->key[n + 2 - p0 + mid];
      is = first ? mid + 1 : is;
      up = first ? up : mid;
    }
  }
  il = n + 1 - p0 + is;
  double sk = sh->key[is], lk = sh->key[il];
  u32 lp = sh->pos[il];
  __syncthreads();  // from here on slots take the place of keys
  if (cnt) {
    u32 ps = A + is * 8, pl = A + il * 8;
    const u32 end = A + S * 8;
#pragma unroll 1
    for (u32 k = 0; k < cnt; ++k) merge_wide_step(sk, lk, lp, ps, pl, end, P - A / 4);
    if (p0 + cnt == n && (ps != end || pl != end + 8)) dev_fail(err, DEV_ERR_INTERNAL, v, p0, 8);  // both lists are used up
  }
  __syncthreads();
  items.weights();
  // in the order of the two lists: neighbouring entries of either are near one another in the list of weights
  for (u32 y = t; y < n; y += NT)
    reinterpret_cast<uint2*>(slots)[(u64)off + sh->pos[y < S ? y : y + 2]] = reinterpret_cast<const uint2*>(sh->key)[y + 1];
  if (t == 0) valid[v] = 1;
}

}  // namespace skw

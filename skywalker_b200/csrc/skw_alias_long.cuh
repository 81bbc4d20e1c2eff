// Table of one weight list that is too long for the registers of a CTA (skw_alias_wide.cuh), by a CTA or by a cluster of them,
// which share it out in chunks: two passes for the largest weight and the total, one in tiles of up to 4096 weights that
// writes the two lists to global memory, and the merge in windows of up to 4096 entries.
// Bound by the latencies of its phases: 221 warp instructions per 32 edges by single CTAs, three an SM, at 41 % of the issue
// slots (some 300 by clusters of eight).  A CTA alone is the whole latency of a list, 0.13 ms for 20,000 weights and 0.5 for 92,000,
// so there is a cluster for each while lists are few (long_team).  16.7 M edges in lists of one length, by one CTA of 1024
// threads and tiles of eight weights a thread before: 16,385 weights 338 -> 265 us, 19,900 341 -> 253, 24,300 330 -> 264,
// 33,000 370 -> 326, 100,000 515 -> 410.
//
// A tile is worked through as a short list is (skw_alias_f64.cuh): weights, masses and the sums inside the tile are
// doubles, all of them exact.  What crosses a tile is a 64-bit integer, since a prefix has up to 62 bits here: a list entry
// is the double relative to its thread's first weight, whose bits (biased by 2^52) are added to the thread's 64-bit base.
// The running weight is counted from the multiple of 2^32 below the tile's base, so that one addition rounds it as the
// conversion of the 64-bit sum would be rounded.  Only a weight of more than 256 buckets has a mass that a double might
// not hold; its thread goes the way of 64-bit integers.  Entries are relative to their chunk, so that no CTA has to know
// the others' sums before it writes its part.
#pragma once
#include <cooperative_groups.h>

#include "skw_alias_f64.cuh"

namespace skw {

constexpr u32 kLongTeam = 8;                          // CTAs a list, at most
constexpr u32 kLongThreads = 256, kLongTile = 4096;  // threads a CTA; weights a tile and entries a merge window, at most

// g(Q) as a double for Q = base + what rel counts from the multiple of 2^32 below base (rel stays below 2^53).
struct LongMass {
  double hi, Wrel, nC, K;
  __device__ __forceinline__ LongMass(u64 base, u64 W, double all, double factor) : nC(all), K(factor) {
    const u32 h = (u32)(base >> 32), dh = (u32)(W >> 32) - h;
    hi = __dmul_rn(u32_to_double(h), 4294967296.0);
    Wrel = dh < (1u << 21) ? __dadd_rn(__dmul_rn(u32_to_double(dh), 4294967296.0), u32_to_double((u32)W)) : -1.0;
  }
  __device__ __forceinline__ double operator()(double rel) const {
    const double g = trunc(__dmul_rn(__dadd_rn(hi, rel), K));
    return rel == Wrel || g > nC ? nC : g;
  }
};

// One list entry, stored if k < cnt: a small (c > 0) with the deficit before it at index is, a large with the excess up to
// and including it at index il; keys at shared address A, positions at P.  D, X: biased and relative to the thread's bases.
__device__ __forceinline__ void put_long_entry(double c, u32 k, u32 cnt, u32 pos, u32 A, u32 P, u64 baseD, u64 baseX, double& D,
                                               double& X, u32& is, u32& il) {
  asm volatile(
      "{\n\t.reg .pred p, in;\n\t.reg .f64 key;\n\t.reg .b64 bits, base;\n\t.reg .b32 i, at;\n\t"
      "setp.gt.f64 p, %4, 0d0000000000000000;\n\t"
      "setp.lt.u32 in, %5, %6;\n\t"
      "@!p sub.rn.f64 %1, %1, %4;\n\t"
      "selp.f64 key, %0, %1, p;\n\t"
      "selp.b64 base, %10, %11, p;\n\t"
      "selp.b32 i, %2, %3, p;\n\t"
      "@p add.rn.f64 %0, %0, %4;\n\t"
      "@p add.u32 %2, %2, 1;\n\t"
      "@!p sub.u32 %3, %3, 1;\n\t"
      "mov.b64 bits, key;\n\t"
      "add.u64 bits, bits, base;\n\t"
      "mad.lo.u32 at, i, 8, %8;\n\t"
      "@in st.shared.u64 [at], bits;\n\t"
      "mad.lo.u32 at, i, 4, %9;\n\t"
      "@in st.shared.u32 [at], %7;\n\t}"
      : "+d"(D), "+d"(X), "+r"(is), "+r"(il)
      : "d"(c), "r"(k), "r"(cnt), "r"(pos), "r"(A), "r"(P), "l"(baseD), "l"(baseX)
      : "memory");
}

// One window of the merge: Sl smalls at index 0 .. Sl with the prefix of the small after them at Sl, Ll = nl - Sl larges
// from index nl + 1 down with the large after them at Sl + 1; keys (8 bytes) and positions (4 bytes) in shared memory.
// Order and outcome as in merge_f64: thread t emits an equal share, a small at the head goes first if its key is not
// above the large's, and what an entry keeps follows from the small list's head after the entry was replaced.
// The slot of an entry that leaves is stored where the next head of its list was read (which nobody needs any more, since
// all threads have read the heads that they begin with), and the slots go out in the order of the two lists, where
// neighbours are near one another in the list of weights: written from the loop they would fall into 32 different sectors.
// All threads of the CTA come here; the caller waits for them before the window is reused.
template <int NT>
__device__ __forceinline__ void merge_long(u32 t, u32 nl, u32 Sl, u64* key, const u32* pos, u64 C, int B, Slot* __restrict__ out) {
  const u32 Ll = nl - Sl;
  const u32 share = (nl + NT - 1) / NT;
  const u32 k0 = min(t * share, nl), k1 = min(k0 + share, nl);
  u32 lo = k0 > Ll ? k0 - Ll : 0, hi = min(k0, Sl);
  while (lo < hi) {  // small mid precedes large k0-1-mid iff its key is not above that large's
    const u32 mid = (lo + hi) >> 1;
    const bool before = key[mid] <= key[nl + 2 - k0 + mid];
    lo = before ? mid + 1 : lo;
    hi = before ? hi : mid;
  }
  const u32 A = (u32)__cvta_generic_to_shared(key), P = (u32)__cvta_generic_to_shared(pos) - A / 2;
  const u32 il = nl + 1 - (k0 - lo), end = A + Sl * 8;
  u32 ps = A + lo * 8, pl = A + il * 8, lp = pos[il];
  u64 sk = key[lo], lk = key[il];
  const float unit = __uint_as_float((u32)(127 - B) << 23);
  __syncthreads();
#pragma unroll 1
  for (u32 k = k0; k < k1; ++k) {
    asm volatile(
        "{\n\t.reg .pred take, more, whole;\n\t.reg .b64 was, next;\n\t.reg .s64 mass;\n\t.reg .b32 at, of, old, bits, alias;\n\t"
        ".reg .f32 prob;\n\t"
        "setp.ne.u32 more, %3, %5;\n\t"
        "setp.le.and.u64 take, %0, %1, more;\n\t"
        "selp.b64 was, %0, %1, take;\n\t"
        "mov.b32 old, %2;\n\t"
        "@take add.u32 %3, %3, 8;\n\t"
        "@!take sub.u32 %4, %4, 8;\n\t"
        "selp.b32 at, %3, %4, take;\n\t"
        "shr.u32 of, at, 1;\n\t"
        "add.u32 of, of, %6;\n\t"
        "ld.shared.u64 next, [at];\n\t"
        "@!take ld.shared.u32 %2, [of];\n\t"
        "@take mov.b64 %0, next;\n\t"
        "@!take mov.b64 %1, next;\n\t"
        "sub.s64 mass, was, %0;\n\t"
        "setp.eq.s64 whole, mass, 0;\n\t"
        "add.s64 mass, mass, %7;\n\t"
        "cvt.rn.f32.s64 prob, mass;\n\t"
        "mul.rn.f32 prob, prob, %8;\n\t"
        "selp.b32 alias, old, %2, whole;\n\t"
        "mov.b32 bits, prob;\n\t"
        "st.shared.v2.b32 [at], {bits, alias};\n\t}"
        : "+l"(sk), "+l"(lk), "+r"(lp), "+r"(ps), "+r"(pl)
        : "r"(end), "r"(P), "l"(C), "f"(unit)
        : "memory");
  }
  __syncthreads();
  for (u32 y = t; y < nl; y += NT)
    reinterpret_cast<uint2*>(out)[pos[y < Sl ? y : y + 2]] = reinterpret_cast<const uint2*>(key)[y + 1];
}

// Shared memory of a CTA: the entries of a tile or of a merge window, the tile's weights, and what is handed around.
struct LongShared {
  u64 key[kLongTile + 2];
  u32 pos[kLongTile + 2];
  int stage[kLongThreads * 17];  // 16 weights a thread, spread by one word a thread
  CtaCoop<(int)kLongThreads>::Words words;
  u64 warp_sum[kLongThreads / 32];
  // of this CTA's chunk, read by the others of the cluster: largest weight, quantised sum, deficit, smalls
  int chunk_top;
  u64 chunk_q, chunk_d;
  u32 chunk_s;
  u64 before_d[kLongTeam + 1];  // deficit and smalls before each chunk
  u32 before_s[kLongTeam + 1];
  u32 bound[32];                   // smalls before the start of each window of a round
};

// Waits for the other CTAs of the cluster, and makes what each wrote before visible to all.
template <u32 CL>
__device__ __forceinline__ void cluster_sync() {
  if constexpr (CL > 1) cooperative_groups::this_cluster().sync();
  else __syncthreads();
}
template <u32 CL, class T>
__device__ __forceinline__ T* cluster_peer(T* mine, u32 rank) {
  if constexpr (CL > 1) return cooperative_groups::this_cluster().map_shared_rank(mine, rank);
  else return mine;
}

// The rank-th of CL CTAs.  (A function of its own: inlined into the loops over the lists it spilled 50 registers a thread.)
// A, P: n keys and positions in global memory, shared by the cluster: a chunk's smalls from its
// front, its larges from its back.
template <u32 CL>
__device__ __noinline__ void build_list_long(u32 rank, u32 v, u32 off, u32 n, const float* __restrict__ w,
                                                   Slot* __restrict__ slots, uint8_t* __restrict__ valid, LongShared* sh,
                                                   u64* A, u32* P, u32* err) {
  constexpr u32 NT = kLongThreads;
  constexpr int EPT = 16;
  const u32 t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const CtaCoop<(int)NT> co(&sh->words, 0);
  const u32 chunk = ((n - 1) / CL / NT + 1) * NT;
  auto chunk_begin = [&](u32 c) { return (u32)min((u64)c * chunk, (u64)n); };
  const u32 cb = chunk_begin(rank), ce = chunk_begin(rank + 1);
  // ---- largest weight; bits of positive floats are ordered as the floats are, others count as zero
  auto usable = [](int x) { return (u32)(x - 1) < 0x7F7FFFFFu ? x : 0; };
  int top = 0;
  for (u32 p = cb; p < ce; p += min(16 * NT, ce - p)) {
    int x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = t + k * NT < ce - p ? __float_as_int(__ldg(w + p + t + k * NT)) : 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) top = max(top, usable(x[k]));
  }
  top = co.template max<0>(top);
  if (t == 0) sh->chunk_top = top;
  cluster_sync<CL>();
  top = GroupCoop<32>().template max<0>(lane < CL ? *cluster_peer<CL>(&sh->chunk_top, lane) : 0);
  if (top == 0) {
    for (u64 p = cb + t; p < ce; p += NT) slots[(u64)off + p] = Slot{-1.0f, (u32)p};
    if (rank == 0 && t == 0) valid[v] = 0;
    return;
  }
  const int B = bucket_bits(n);
  const u64 C = (u64)1 << B, nC = (u64)n << B;
  // lists whose largest weight is below 2^-87 are scaled up, so that zeros and denormals quantise to 0
  const float scale = top < (40 << 23) ? 18446744073709551616.0f : 1.0f;
  const u64 shift = (u64)(1022 + B - (__float_as_int(__int_as_float(top) * scale) >> 23)) << 52;
  auto quantised = [&](int x) {
    const int b = usable(__float_as_int(__int_as_float(x) * scale));
    const double y = __longlong_as_double((long long)((u64)(u32)b * (1u << 29) + shift));
    return __dsub_rn(__dadd_rz(y, kTwo52), kTwo52);
  };
  // ---- total, and what is before this chunk
  u64 W = 0, Qc = 0;
  for (u32 p = cb; p < ce; p += min(16 * NT, ce - p)) {
    int x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = t + k * NT < ce - p ? __float_as_int(__ldg(w + p + t + k * NT)) : 0;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) s = __dadd_rn(s, quantised(x[k]));
    W += (u64)s;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) W += __shfl_xor_sync(0xFFFFFFFFu, W, o);
  if (lane == 0) sh->warp_sum[warp] = W;
  __syncthreads();
  if (t == 0) {
    u64 q = 0;
#pragma unroll
    for (u32 x = 0; x < NT / 32; ++x) q += sh->warp_sum[x];
    sh->chunk_q = q;
  }
  cluster_sync<CL>();
  W = lane < CL ? *cluster_peer<CL>(&sh->chunk_q, lane) : 0;
  Qc = lane < rank ? W : 0;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    W += __shfl_xor_sync(0xFFFFFFFFu, W, o);
    Qc += __shfl_xor_sync(0xFFFFFFFFu, Qc, o);
  }
  const double K = mass_factor(n, B, W), bucket = pow2d(B);
  // ---- lists
  const u32 sA = (u32)__cvta_generic_to_shared(sh->key), sP = (u32)__cvta_generic_to_shared(sh->pos);
  u64 Dc = 0;  // of the chunk, before the tile: deficit, smalls
  u32 Sc = 0;
  // tiles of equal size: a last one of a few weights would take as many instructions as a full one
  const u32 tiles = (ce - cb + kLongTile - 1) / kLongTile;
  const u32 tile = tiles ? ((ce - cb - 1) / tiles / NT + 1) * NT : 0;
  constexpr int CH = 2;
#define SKW_EACH(k)                                        \
  _Pragma("unroll") for (int b_ = 0; b_ < EPT; b_ += CH) { \
    if ((u32)b_ >= ept) break;                             \
    _Pragma("unroll") for (int k = b_; k < b_ + CH; ++k)
#define SKW_EACH_END }
  for (u32 base = cb; base < ce; base += min(tile, ce - base)) {
    const u32 here = min(tile, ce - base);
    const u32 ept = (here + NT - 1) / NT;
    const u32 p0 = min(t * ept, here), cnt = min(ept, here - p0);  // this thread's elements of the tile
    const u32 over = min((ept + CH - 1) / CH * CH, (u32)EPT) - cnt;
    const u32 per = ept & 1 ? 0u : 0xFFFFFFFFu / ept + 1;  // i / ept as a multiplication (i < 4096)
    const int* mine = sh->stage + t * (ept | 1);
    double c[EPT];
    {
      int x[EPT];
#pragma unroll
      for (int k = 0; k < EPT; ++k) x[k] = t + k * NT < here ? __float_as_int(__ldg(w + base + t + k * NT)) : 0;
      SKW_EACH(k) {
        const u32 i = t + k * NT;
        if (i < here) sh->stage[i + __umulhi(i, per)] = x[k];
      }
      SKW_EACH_END
    }
    __syncthreads();
    double Q = 0.0, all;
    SKW_EACH(k) {
      c[k] = quantised((u32)k < cnt ? mine[k] : 0);
      Q = __dadd_rn(Q, c[k]);
    }
    SKW_EACH_END
    co.scan(Q, all);
    const LongMass mass(Qc, W, __ull2double_rn(nC), K);
    const double first = __dadd_rn(u32_to_double((u32)Qc), Q);  // the running weight at the thread's first element
    Qc += (u64)all;
    double rel = first, g = mass(rel), D = 0.0, tD;
    const u64 net = (u64)g - (u64)(base + p0) * C;  // excess minus deficit there
    u32 s = 0, tS, giant = 0;
    SKW_EACH(k) {
      rel = __dadd_rn(rel, c[k]);
      const double gn = mass(rel);
      c[k] = __dsub_rn(bucket, __dsub_rn(gn, g));  // what a small lacks, minus what a large has too much
      g = gn;
      giant = max(giant, (u32)__double2hiint(c[k]));
      count_small(c[k], D, s);
    }
    SKW_EACH_END
    D = __dsub_rn(D, __dmul_rn((double)over, bucket));
    s -= over;
    co.scan(D, s, tD, tS);
    // the bits of a double biased by 2^52, plus one of these, are a list entry
    const u64 baseD = Dc + (u64)D, baseX = baseD + net;
    u32 is = s, il = here - 1 - (p0 - s);
    if (giant < 0xC2F00000u) {  // no excess of 2^48 or more: all sums of a thread stay below 2^52
      double Dr = kTwo52, Xr = kTwo52;
      const u64 bias = (u64)kBiasHi << 32;
      SKW_EACH(k) { put_long_entry(c[k], k, cnt, base + p0 + k, sA, sP, baseD - bias, baseX - bias, Dr, Xr, is, il); }
      SKW_EACH_END
    } else {
      u64 d = baseD, x = baseX, gi = (u64)mass(first);
      rel = first;
#pragma unroll 1
      for (u32 k = 0; k < cnt; ++k) {
        rel = __dadd_rn(rel, quantised(mine[k]));
        const u64 gn = (u64)mass(rel), m = gn - gi;
        gi = gn;
        const bool small = m < C;
        if (!small) x += m - C;
        const u32 i = small ? is : il;
        sh->key[i] = small ? d : x;
        sh->pos[i] = base + p0 + k;
        if (small) d += C - m;
        is += small ? 1u : 0u;
        il -= small ? 0u : 1u;
      }
    }
    __syncthreads();
    // a thread's entries alone would go out as scattered stores
    const u32 lb = ce - 1 - (base - cb - Sc);  // the tile's first large goes here, the others below it
    for (u32 y = t; y < here; y += NT) {
      const u32 to = y < tS ? cb + Sc + y : lb - (here - 1 - y);
      A[to] = sh->key[y];
      P[to] = sh->pos[y];
    }
    // (the next tile's entries are three barriers away)
    Dc += (u64)tD;
    Sc += tS;
  }
#undef SKW_EACH
#undef SKW_EACH_END
  if (t == 0) {
    sh->chunk_d = Dc;
    sh->chunk_s = Sc;
  }
  cluster_sync<CL>();
  if (t == 0) {
    u64 d = 0;
    u32 s = 0;
#pragma unroll
    for (u32 c = 0; c < CL; ++c) {
      sh->before_d[c] = d;
      sh->before_s[c] = s;
      d += *cluster_peer<CL>(&sh->chunk_d, c);
      s += *cluster_peer<CL>(&sh->chunk_s, c);
    }
    sh->before_d[CL] = d;
    sh->before_s[CL] = s;
  }
  __syncthreads();
  const u32 S = sh->before_s[CL], L = n - S;
  if (L == 0) {  // mass conservation guarantees a large
    if (t == 0) dev_fail(err, DEV_ERR_INTERNAL, v, L, 7);
    for (u64 p = cb + t; p < ce; p += NT) slots[(u64)off + p] = Slot{1.0f, (u32)p};
    if (rank == 0 && t == 0) valid[v] = 1;
    return;
  }
  // ---- merge: this CTA's windows of the merged order.  Small i and large j by their chunks (other CTAs wrote most of
  // them, so they are read from L2):
  auto larges_before = [&](u32 c) { return chunk_begin(c) - sh->before_s[c]; };
  auto small_key = [&](u32 i) {
    u32 c = 0;
    while (c + 1 < CL && i >= sh->before_s[c + 1]) ++c;
    return __ldcg(A + chunk_begin(c) + (i - sh->before_s[c])) + sh->before_d[c];
  };
  auto large_key = [&](u32 j) {
    u32 c = 0;
    while (c + 1 < CL && j >= larges_before(c + 1)) ++c;
    return __ldcg(A + chunk_begin(c + 1) - 1 - (j - larges_before(c))) + sh->before_d[c];
  };
  const u32 each = (n - 1) / kLongTile / CL + 1, size = (n - 1) / (each * CL) + 1;  // windows a CTA, entries a window
  for (u32 w0 = rank * each; w0 < (rank + 1) * each; w0 += 31) {  // a round of cnt windows needs cnt + 1 boundaries
    const u32 cnt = min(31u, (rank + 1) * each - w0);
    __syncthreads();
    for (u32 x = warp; x <= cnt; x += NT / 32) {  // a warp finds one boundary, with 32 probes a step
      const u32 k0 = (u32)min((u64)(w0 + x) * size, (u64)n);
      u32 lo = k0 > L ? k0 - L : 0, hi = min(k0, S);
      while (lo < hi) {
        const u32 step = (hi - lo + 31) / 32;
        const u64 mid = (u64)lo + (u64)lane * step;
        // small mid precedes large k0-1-mid iff its key is not above that large's
        const bool before = mid < hi && small_key((u32)mid) <= large_key(k0 - 1 - (u32)mid);
        const u32 many = __popc(__ballot_sync(0xFFFFFFFFu, before));
        if (many == 0) break;
        hi = (u32)min((u64)lo + (u64)many * step, (u64)hi);
        lo += (many - 1) * step + 1;
      }
      if (lane == 0) sh->bound[x] = lo;
    }
    __syncthreads();
    for (u32 x = 0; x < cnt; ++x) {
      const u32 k0 = (u32)min((u64)(w0 + x) * size, (u64)n), k1 = (u32)min((u64)k0 + size, (u64)n);
      const u32 i0 = sh->bound[x], i1 = sh->bound[x + 1], j0 = k0 - i0, j1 = k1 - i1;
      const u32 Sl = i1 - i0, nl = k1 - k0;
      if (nl == 0) break;
#pragma unroll 1
      for (u32 c = 0; c < CL; ++c) {  // the window's entries and the one after either list, chunk by chunk
        const u64 d = sh->before_d[c];
        const u32 b = chunk_begin(c), e = chunk_begin(c + 1);
        const u32 sb = sh->before_s[c], se = sh->before_s[c + 1], lb = b - sb, le = e - se;
        for (u32 i = max(i0, sb) + t; i < min(i1 + 1, se); i += NT) {
          sh->key[i - i0] = __ldcg(A + b + (i - sb)) + d;
          sh->pos[i - i0] = __ldcg(P + b + (i - sb));
        }
        for (u32 j = max(j0, lb) + t; j < min(j1 + 1, le); j += NT) {
          sh->key[nl + 1 - (j - j0)] = __ldcg(A + e - 1 - (j - lb)) + d;
          sh->pos[nl + 1 - (j - j0)] = __ldcg(P + e - 1 - (j - lb));
        }
      }
      if (t == 0 && i1 == S) {  // behind the last small: the total deficit
        sh->key[Sl] = sh->before_d[CL];
        sh->pos[Sl] = 0;
      }
      if (t == 0 && j1 == L) {
        sh->key[Sl + 1] = ~0ull;
        sh->pos[Sl + 1] = 0;
      }
      __syncthreads();
      merge_long<(int)NT>(t, nl, Sl, sh->key, sh->pos, C, B, slots + off);
      __syncthreads();
    }
  }
  if (rank == 0 && t == 0) valid[v] = 1;
}

}  // namespace skw

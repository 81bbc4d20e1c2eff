// Table of one weight list that is too long for the registers of a CTA (skw_alias_f64.cuh): two passes for the largest
// weight and the total, one in tiles of eight weights a thread that writes the two lists, and the merge.
//
// Weights are quantised as doubles (the float's bits in place, see skw_alias_f64.cuh) and summed as doubles inside a warp,
// where the sums are exact; what crosses a warp, masses and prefixes are 64-bit integers, since a prefix has up to 62
// bits here.  The running weight of a thread is a double relative to its warp's base, and one addition to the base's
// multiple of 2^32 rounds it as the conversion of the 64-bit sum would be rounded.
// Bound by instruction issue and, in the merge, by the latency of shared memory: 8.2 warp instructions an edge at 43 % of the
// issue slots; 254 lists of 26,500 weights 340 us.
#pragma once
#include "skw_alias_f64.cuh"

namespace skw {

__device__ __forceinline__ double u32_to_double(u32 x) { return __dsub_rn(__hiloint2double((int)kBiasHi, (int)x), kTwo52); }

// g(Q) for Q = base + what rel counts from the multiple of 2^32 below base.
struct MassAt {
  double hi, Wrel;
  __device__ __forceinline__ MassAt(u64 base, u64 W) {
    const u32 h = (u32)(base >> 32), dh = (u32)(W >> 32) - h;
    hi = __dmul_rn(u32_to_double(h), 4294967296.0);
    Wrel = dh < (1u << 20) ? __dadd_rn(__dmul_rn(u32_to_double(dh), 4294967296.0), u32_to_double((u32)W)) : -1.0;
  }
  __device__ __forceinline__ u64 operator()(double rel, double K, u64 nC) const {
    const u64 g = __double2ull_rz(__dmul_rn(__dadd_rn(hi, rel), K));
    return rel == Wrel || g > nC ? nC : g;
  }
};

// Cross-thread words of a CTA of NT threads.
template <int NT>
struct LongWords {
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

// One window of the merge: Sl smalls at index 0 .. Sl with the prefix of the small after them at Sl, Ll = nl - Sl larges
// from index nl + 1 down with the large after them at Sl + 1; keys (8 bytes) at shared address A, positions (4 bytes) at P.
// Order and outcome as in merge_f64: thread t emits an equal share, a small at the head goes first if its key is not
// above the large's, and what an entry keeps follows from the small list's head after the entry was replaced.
template <int NT>
__device__ __forceinline__ void merge_long(u32 t, u32 nl, u32 Sl, u32 A, u32 P, u64 C, int B, Slot* __restrict__ out) {
  const u32 Ll = nl - Sl;
  const u32 share = (nl + NT - 1) / NT;
  const u32 k0 = min(t * share, nl), k1 = min(k0 + share, nl);
  if (k0 >= k1) return;
  auto key = [&](u32 i) {
    u64 x;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(x) : "r"(A + i * 8) : "memory");
    return x;
  };
  auto pos = [&](u32 i) {
    u32 x;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(P + i * 4) : "memory");
    return x;
  };
  u32 lo = k0 > Ll ? k0 - Ll : 0, hi = min(k0, Sl);
  while (lo < hi) {  // small mid precedes large k0-1-mid iff its key is not above that large's
    const u32 mid = (lo + hi) >> 1;
    const bool before = key(mid) <= key(nl + 2 - k0 + mid);
    lo = before ? mid + 1 : lo;
    hi = before ? hi : mid;
  }
  u32 is = lo, il = nl + 1 - (k0 - lo);
  u64 sk = key(is), lk = key(il);
  u32 sp = pos(is), lp = pos(il);
  const float unit = __uint_as_float((u32)(127 - B) << 23);
#pragma unroll 4
  for (u32 k = k0; k < k1; ++k) {
    asm volatile(
        "{\n\t.reg .pred take, more, whole;\n\t.reg .b64 was, to;\n\t.reg .s64 mass;\n\t.reg .b32 p, i, at, bits, alias;\n\t"
        ".reg .f32 prob;\n\t"
        "setp.ne.u32 more, %4, %6;\n\t"
        "setp.le.and.u64 take, %0, %1, more;\n\t"
        "selp.b64 was, %0, %1, take;\n\t"
        "selp.b32 p, %2, %3, take;\n\t"
        "@take add.u32 %4, %4, 1;\n\t"
        "@!take sub.u32 %5, %5, 1;\n\t"
        "selp.b32 i, %4, %5, take;\n\t"
        "mad.lo.u32 at, i, 8, %7;\n\t"
        "@take ld.shared.u64 %0, [at];\n\t"
        "@!take ld.shared.u64 %1, [at];\n\t"
        "mad.lo.u32 at, i, 4, %8;\n\t"
        "@take ld.shared.u32 %2, [at];\n\t"
        "@!take ld.shared.u32 %3, [at];\n\t"
        "sub.s64 mass, was, %0;\n\t"
        "setp.eq.s64 whole, mass, 0;\n\t"
        "add.s64 mass, mass, %9;\n\t"
        "cvt.rn.f32.s64 prob, mass;\n\t"
        "mul.rn.f32 prob, prob, %10;\n\t"
        "selp.b32 alias, p, %3, whole;\n\t"
        "mov.b32 bits, prob;\n\t"
        "mad.wide.u32 to, p, 8, %11;\n\t"
        "st.global.v2.b32 [to], {bits, alias};\n\t}"
        : "+l"(sk), "+l"(lk), "+r"(sp), "+r"(lp), "+r"(is), "+r"(il)
        : "r"(Sl), "r"(A), "r"(P), "l"(C), "f"(unit), "l"(out)
        : "memory");
  }
}

// Shared memory of build_list_long: a merge window of CAP entries, then the tile's weights, transposed so that neither writing nor reading them meets the same bank twice.
template <int NT, int CAP>
struct LongShared {
  u64 key[CAP + 2];
  u32 pos[CAP + 2];
  int stage[8][NT + 4];
  LongWords<NT> words;
};

// The lists (n + 2 entries) are in global memory at A, P and are merged through windows of CAP entries.
template <int NT, int CAP>
__device__ __forceinline__ void build_list_long(u32 v, u32 off, u32 n, const float* __restrict__ w, Slot* __restrict__ slots,
                                                uint8_t* __restrict__ valid, LongShared<NT, CAP>* sh, u64* A, u32* P,
                                                u32* err) {
  constexpr u32 NW = NT / 32, kTile = NT * 8;
  const u32 t = threadIdx.x, lane = t & 31, warp = t >> 5;
  LongWords<NT>& words = sh->words;
  const GroupCoop<32> wc;
  // ---- largest weight; bits of positive floats are ordered as the floats are, others count as zero
  auto usable = [](int x) { return (u32)(x - 1) < 0x7F7FFFFFu ? x : 0; };
  int top = 0;
  for (u32 p = t; p < n; p += kTile) {
    int x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = n - p > k * NT ? __float_as_int(__ldg(w + p + k * NT)) : 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) top = max(top, usable(x[k]));
    if (n - p <= kTile) break;  // (p + kTile may pass 2^32)
  }
  top = wc.max<0>(top);
  if (lane == 0) words.s[warp] = (u32)top;
  __syncthreads();
  top = wc.max<0>(lane < NW ? (int)words.s[lane] : 0);
  if (top == 0) {
    for (u64 p = t; p < n; p += NT) slots[(u64)off + p] = Slot{-1.0f, (u32)p};
    if (t == 0) valid[v] = 0;
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
  // ---- total
  u64 W = 0;
  for (u32 p = t; p < n; p += kTile) {
    int x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = n - p > k * NT ? __float_as_int(__ldg(w + p + k * NT)) : 0;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s = __dadd_rn(s, quantised(x[k]));
    W += (u64)s;
    if (n - p <= kTile) break;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) W += __shfl_xor_sync(0xFFFFFFFFu, W, o);
  if (lane == 0) words.d[warp] = W;
  __syncthreads();
  W = lane < NW ? words.d[lane] : 0;
#pragma unroll
  for (int o = 16; o; o >>= 1) W += __shfl_xor_sync(0xFFFFFFFFu, W, o);
  const double K = mass_factor(n, B, W);
  // ---- lists
  u64 Qc = 0, Dc = 0;  // before the tile: quantised weight, deficit, smalls
  u32 Sc = 0;
  for (u32 base = 0;; base += kTile) {
    const u32 here = min(kTile, n - base);
    const u32 ept = (here + NT - 1) / NT;
    const u32 p0 = min(t * ept, here), cnt = min(ept, here - p0);  // this thread's elements of the tile
    const u32 magic = 0xFFFFFFFFu / ept + 1;                       // i / ept as a multiplication (ept > 1)
    int x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = t + k * NT < here ? __float_as_int(__ldg(w + base + t + k * NT)) : 0;
    // (the last readers of the stage are two barriers away)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const u32 i = t + k * NT, who = ept == 1 ? i : __umulhi(i, magic);
      if (i < here) sh->stage[i - who * ept][who] = x[k];
    }
    __syncthreads();
    double q[8], before = 0.0, all;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q[k] = 0.0;
      if ((u32)k < cnt) q[k] = quantised(sh->stage[k][t]);
      before = __dadd_rn(before, q[k]);
    }
    wc.scan(before, all);
    if (lane == 0) words.q[warp] = (u64)all;
    __syncthreads();
    u64 tile_q, wq = warp_scan_u64(lane < NW ? words.q[lane] : 0, lane, tile_q);
    wq = Qc + __shfl_sync(0xFFFFFFFFu, wq, warp);  // before this warp
    Qc += tile_q;
    const MassAt mass(wq, W);
    double rel = __dadd_rn(u32_to_double((u32)wq), before);
    u64 g = mass(rel, K, nC);
    u64 Z = g - (u64)(base + p0) * C;  // excess minus deficit before this thread
    u64 m[8], D = 0;
    u32 s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      m[k] = C;
      if ((u32)k < cnt) {
        rel = __dadd_rn(rel, q[k]);
        const u64 gn = mass(rel, K, nC);
        m[k] = gn - g;
        g = gn;
        if (m[k] < C) {
          D += C - m[k];
          ++s;
        }
      }
    }
    u64 wd, inc;
    {
      u64 d_incl = D;
      u32 s_incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u64 y = __shfl_up_sync(0xFFFFFFFFu, d_incl, o);
        const u32 z = __shfl_up_sync(0xFFFFFFFFu, s_incl, o);
        if (lane >= (u32)o) {
          d_incl += y;
          s_incl += z;
        }
      }
      if (lane == 31) {
        words.d[warp] = d_incl;
        words.s[warp] = s_incl;
      }
      D = d_incl - D;
      s = s_incl - s;
    }
    __syncthreads();
    {
      u64 tile_d;
      wd = warp_scan_u64(lane < NW ? words.d[lane] : 0, lane, tile_d);
      u32 sw = lane < NW ? words.s[lane] : 0, s_incl = sw;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 z = __shfl_up_sync(0xFFFFFFFFu, s_incl, o);
        if (lane >= (u32)o) s_incl += z;
      }
      D += Dc + __shfl_sync(0xFFFFFFFFu, wd, warp);
      s += Sc + __shfl_sync(0xFFFFFFFFu, s_incl - sw, warp);
      Dc += tile_d;
      inc = __shfl_sync(0xFFFFFFFFu, (u64)s_incl, 31);
    }
    // Next entries of this thread in the two lists.  They are laid out in shared memory first (the tile's smalls from the
    // front, its larges from the back) and copied out in order: a thread's entries alone would go out as scattered 8-byte
    // stores.
    static_assert(CAP >= (int)kTile, "the merge window doubles as the tile's staging area");
    u32 is = s - Sc, il = here - 1 - (p0 - is);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if ((u32)k < cnt) {
        const bool small = m[k] < C;
        const u64 e = m[k] - C;
        Z += e;
        const u64 key = small ? D : D + Z;  // deficit before a small, excess up to and including a large
        const u32 i = small ? is : il;
        sh->key[i] = key;
        sh->pos[i] = base + p0 + k;
        D -= small ? e : 0;
        is += small ? 1u : 0u;
        il -= small ? 0u : 1u;
      }
    }
    __syncthreads();
    const u32 ts = (u32)inc;  // smalls of this tile; the larges before it are base - Sc
    for (u32 y = t; y < here; y += NT) {
      const u64 to = y < ts ? (u64)Sc + y : (u64)n + 1 - (base - Sc) - (here - 1 - y);
      A[to] = sh->key[y];
      P[to] = sh->pos[y];
    }
    // (the next tile's entries are three barriers away)
    Sc += (u32)inc;
    if (n - base <= kTile) break;
  }
  const u32 S = Sc, L = n - S;
  if (t == 0) {
    A[S] = Dc;  // what the last small exceeds, and what stands behind the last large
    P[S] = 0;
    A[S + 1] = ~0ull;
    P[S + 1] = 0;
  }
  __syncthreads();
  if (L == 0) {  // mass conservation guarantees a large
    if (t == 0) dev_fail(err, DEV_ERR_INTERNAL, v, L, 7);
    for (u64 p = t; p < n; p += NT) slots[(u64)off + p] = Slot{1.0f, (u32)p};
    if (t == 0) valid[v] = 1;
    return;
  }
  const u32 sA = (u32)__cvta_generic_to_shared(sh->key), sP = (u32)__cvta_generic_to_shared(sh->pos);
  // the merged order in windows of CAP: each window's slices of the two lists (and the entry after either) come into
  // shared memory with coalesced copies
  u32* bnd = reinterpret_cast<u32*>(sh->stage);  // smalls before the start of each window of a round
  const u32 nwin = (n + CAP - 1) / CAP;
  for (u32 w0 = 0; w0 < nwin; w0 += NT - 1) {  // a round of cnt windows needs cnt + 1 boundaries
    const u32 cnt = min((u32)NT - 1, nwin - w0);
    __syncthreads();
    if (t <= cnt) {  // one bisection per window boundary, all in parallel
      const u32 k0 = (u32)min((u64)(w0 + t) * CAP, (u64)n);
      u32 lo = k0 > L ? k0 - L : 0, hi = min(k0, S);
      while (lo < hi) {
        const u32 mid = lo + ((hi - lo) >> 1);
        const bool before = A[mid] <= A[n + 2 - k0 + mid];
        lo = before ? mid + 1 : lo;
        hi = before ? hi : mid;
      }
      bnd[t] = lo;
    }
    __syncthreads();
    for (u32 wi = 0; wi < cnt; ++wi) {
      const u32 k0 = (w0 + wi) * (u32)CAP, k1 = (u32)min((u64)k0 + CAP, (u64)n);
      const u32 i0 = bnd[wi], i1 = bnd[wi + 1], j0 = k0 - i0, j1 = k1 - i1;
      const u32 Sl = i1 - i0, Ll = j1 - j0, nl = Sl + Ll;
      for (u32 y = t; y <= Sl; y += NT) {
        sh->key[y] = A[i0 + y];
        sh->pos[y] = P[i0 + y];
      }
      for (u32 y = t; y <= Ll; y += NT) {  // large j0 + y
        sh->key[nl + 1 - y] = A[n + 1 - j0 - y];
        sh->pos[nl + 1 - y] = P[n + 1 - j0 - y];
      }
      __syncthreads();
      merge_long<NT>(t, nl, Sl, sA, sP, C, B, slots + off);
      __syncthreads();
    }
  }
  if (t == 0) valid[v] = 1;
}

}  // namespace skw

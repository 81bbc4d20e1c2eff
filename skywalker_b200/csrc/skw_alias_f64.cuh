// Table of one weight list of at most 4096 entries, in double precision.
//
// The construction rule works on integers below 2^53 for such lists (bucket 2^40, n <= 2^12 of them), so a double
// holds every one of them exactly and one FP64 instruction does what two or three integer ones did: an addition,
// a comparison or a difference of 64-bit values is one DADD or DSETP.  The integer pipe bound the 64-bit version
// (busy 66-76 % of the time at 8.4 warp instructions an edge, the FP64 pipe 1 %).  The bits of the table are those
// of the integer rule:
//   quantised weight   the float's bits times 2^29 plus a constant ARE the double w * 2^(39 - e) (e = exponent of the
//                      largest weight): one multiply-add; adding 2^52 towards zero and taking it off truncates
//   cumulative mass    g = trunc(Q * K): the product rounded once, truncated by the same addition of 2^52, and kept
//                      with that bias since only differences are used.  Q * K never exceeds n * 2^40 for Q < W
//                      (W <= 2^52, so 1 - 1/W outweighs the two roundings); Q == W is n * 2^40 by definition
//   list entry         a prefix p biased to 2^52 + p has p itself in its low 52 bits; the 12 bits above, which
//                      always hold the same exponent, carry the position instead: 64 bits an entry
//
// Shape: NT cooperating threads (a group of lanes, a warp or a CTA) own EPT consecutive weights each, so a whole
// list is one tile in registers: loaded once, quantised once, two scans, one merge.
#pragma once
#include "skw_alias_math.cuh"

namespace skw {

constexpr u32 kF64Max = 4096;                  // longest list: positions have 12 bits, sums stay below 2^52
constexpr double kTwo52 = 4503599627370496.0;  // 2^52
constexpr double kBucket = 1099511627776.0;    // 2^40, the bucket of every list of up to 2^22 weights
constexpr u32 kBiasHi = 0x43300000u;           // high word of 2^52

__device__ __forceinline__ double u32_to_double(u32 x) { return __dsub_rn(__hiloint2double((int)kBiasHi, (int)x), kTwo52); }
__device__ __forceinline__ uint2 list_entry(double key, u32 pos) {
  return make_uint2((u32)__double2loint(key), (u32)__double2hiint(key) + ((pos << 20) - kBiasHi));
}

// Cooperation inside a group of G lanes of one warp (G = 1, 2, 4 ... 32).  Groups of a warp work on different
// vertices and may diverge, so every shuffle names only the lanes of its own group.
template <int G>
struct GroupCoop {
  static constexpr int NT = G;
  u32 mask, t;
  __device__ __forceinline__ GroupCoop() {
    const u32 lane = threadIdx.x & 31;
    t = lane & (G - 1);
    mask = G == 32 ? 0xFFFFFFFFu : (((1u << G) - 1u) << (lane & ~(u32)(G - 1)));
  }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  template <int USE>
  __device__ __forceinline__ int max(int v) const {
    if (G == 32) return __reduce_max_sync(0xFFFFFFFFu, v);
#pragma unroll
    for (int o = G / 2; o; o >>= 1) v = ::max(v, __shfl_xor_sync(mask, v, o, G));
    return v;
  }
  // v becomes the exclusive prefix over the group, total the group's sum
  __device__ __forceinline__ void scan(double& v, double& total) const {
    double inc = v;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const double x = __shfl_up_sync(mask, inc, o, G);
      if (t >= (u32)o) inc += x;
    }
    total = __shfl_sync(mask, inc, G - 1, G);
    v = inc - v;
  }
  __device__ __forceinline__ void scan(double& v, u32& c, double& total, u32& count) const {
    double inc = v;
    u32 ic = c;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const double x = __shfl_up_sync(mask, inc, o, G);
      const u32 y = __shfl_up_sync(mask, ic, o, G);
      if (t >= (u32)o) {
        inc += x;
        ic += y;
      }
    }
    total = __shfl_sync(mask, inc, G - 1, G);
    count = __shfl_sync(mask, ic, G - 1, G);
    v = inc - v;
    c = ic - c;
  }
};

// Cooperation inside NTHREADS threads of a CTA of 256, the part-th such part of it.  Every reduction has its own words of
// shared memory, so each takes one barrier; the warps all scan the (at most 32) warp totals themselves instead of waiting
// for one that does.
template <int NTHREADS>
struct CtaCoop {
  static constexpr int NT = NTHREADS, NW = NTHREADS / 32;
  struct Words {
    double q[NW], d[NW];
    u32 s[NW];
    int m[2][NW];
  };
  u32 t;
  Words* sh;
  // Barrier of this part (0 is the CTA's own).  Parts of different sizes have different ones: while one part is still at a
  // list, another may have gone on to smaller parts, and a barrier has one thread count at a time.
  u32 bar;
  __device__ __forceinline__ CtaCoop(Words* words, u32 part)
      : t(threadIdx.x % NTHREADS), sh(words), bar(256 / NTHREADS + part) {}
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(NTHREADS) : "memory"); }
  template <int USE>
  __device__ __forceinline__ int max(int v) const {
    v = __reduce_max_sync(0xFFFFFFFFu, v);
    if ((t & 31) == 0) sh->m[USE][t >> 5] = v;
    sync();
    return __reduce_max_sync(0xFFFFFFFFu, sh->m[USE][(t & 31) < NW ? (t & 31) : 0]);
  }
  __device__ __forceinline__ void scan(double& v, double& total) const {
    const GroupCoop<32> w;
    double part = v, sum;
    w.scan(part, sum);
    if ((t & 31) == 0) sh->q[t >> 5] = sum;
    sync();
    double before = (t & 31) < NW ? sh->q[t & 31] : 0.0;
    w.scan(before, total);
    v = part + __shfl_sync(0xFFFFFFFFu, before, t >> 5);
  }
  __device__ __forceinline__ void scan(double& v, u32& c, double& total, u32& count) const {
    const GroupCoop<32> w;
    double part = v, sum;
    u32 pc = c, sc;
    w.scan(part, pc, sum, sc);
    if ((t & 31) == 0) {
      sh->d[t >> 5] = sum;
      sh->s[t >> 5] = sc;
    }
    sync();
    double before = (t & 31) < NW ? sh->d[t & 31] : 0.0;
    u32 bc = (t & 31) < NW ? sh->s[t & 31] : 0u;
    w.scan(before, bc, total, count);
    v = part + __shfl_sync(0xFFFFFFFFu, before, t >> 5);
    c = pc + __shfl_sync(0xFFFFFFFFu, bc, t >> 5);
  }
};

// The steps below are written in PTX: every conditional update is one predicated instruction there, where the
// compiler's selects and branches came out at twice the instructions (merge 65 -> 32, list entry 22 -> 11 per weight).

// Deficit c > 0 of a small goes into the sum D and the count s.
__device__ __forceinline__ void count_small(double c, double& D, u32& s) {
  asm("{\n\t.reg .pred p;\n\t"
      "setp.gt.f64 p, %2, 0d0000000000000000;\n\t"
      "@p add.rn.f64 %0, %0, %2;\n\t"
      "@p add.u32 %1, %1, 1;\n\t}"
      : "+d"(D), "+r"(s)
      : "d"(c));
}
// One list entry, stored if k < cnt: a small (c > 0) with the deficit before it at ps, a large with the excess up to
// and including it at pl.  D, X: the running prefixes, biased; tag: position of the thread's first weight << 20,
// less the bias.
__device__ __forceinline__ void put_entry(double c, u32 k, u32 cnt, u32 tag, double& D, double& X, u32& ps, u32& pl) {
  asm volatile(
      "{\n\t.reg .pred p, in;\n\t.reg .f64 key;\n\t.reg .b32 lo, hi, at;\n\t"
      "setp.gt.f64 p, %4, 0d0000000000000000;\n\t"
      "setp.lt.u32 in, %5, %6;\n\t"
      "@!p sub.rn.f64 %1, %1, %4;\n\t"
      "selp.f64 key, %0, %1, p;\n\t"
      "selp.b32 at, %2, %3, p;\n\t"
      "@p add.rn.f64 %0, %0, %4;\n\t"
      "@p add.u32 %2, %2, 8;\n\t"
      "@!p sub.u32 %3, %3, 8;\n\t"
      "mov.b64 {lo, hi}, key;\n\t"
      "add.u32 hi, hi, %7;\n\t"
      "@in st.shared.v2.b32 [at], {lo, hi};\n\t}"
      : "+d"(D), "+d"(X), "+r"(ps), "+r"(pl)
      : "d"(c), "r"(k), "r"(cnt), "r"(tag + (k << 20))
      : "memory");
}
__device__ __forceinline__ double shared_key(u32 at) {
  double key;
  asm volatile(
      "{\n\t.reg .b32 lo, hi;\n\t"
      "ld.shared.v2.b32 {lo, hi}, [%1];\n\t"
      "lop3.b32 hi, hi, 0xFFFFF, 0x43300000, 0xEA;\n\t"
      "mov.b64 %0, {lo, hi};\n\t}"
      : "=d"(key)
      : "r"(at)
      : "memory");
  return key;
}
__device__ __forceinline__ u32 shared_pos(u32 at) {
  u32 hi;
  asm volatile("ld.shared.u32 %0, [%1+4];" : "=r"(hi) : "r"(at) : "memory");
  return hi >> 20;
}

// The sweep as a merge (see the merge-path builders).  List of n + 1 entries from shared address A on: S smalls, each
// with the deficit before it; the total deficit; n - S larges from the back.  Small i precedes large j iff its key is
// not above the large's.  Thread t emits an equal share of the merged order
// into the list's slots in shared memory: stored where they belong in global memory, the entries of a warp would fall
// into 32 different sectors, which took longer than everything else in this loop.
// A small at the head keeps what the next small's prefix exceeds its own by less than a bucket; a large that leaves
// keeps a bucket less what the prefix of the small at the head exceeds its own by, and is topped up by the large
// behind it.  Both need the head of the small list AFTER the entry that left has been replaced, and the alias is the
// head of the large list after that, whether a small or a large left.  Once every small is placed the small list's
// head is the total deficit, which the last larges' prefix equals: their mass comes out as exactly one bucket (a
// small's never does), and such a large keeps its bucket for itself.
template <int NT>
__device__ __forceinline__ void merge_f64(u32 t, u32 n, u32 S, u32 A, u32 out, u32 v, u32* err) {
  const u32 L = n - S;
  const u32 share = (n + NT - 1) / NT;
  const u32 k0 = min(t * share, n), k1 = min(k0 + share, n);
  if (k0 >= k1) return;
  u32 lo = k0 > L ? k0 - L : 0, hi = min(k0, S);
  const u32 larges = A + (n - k0 + 1) * 8;  // entry of large k0 - 1
  while (lo < hi) {
    const u32 mid = (lo + hi) >> 1;
    const bool before = shared_key(A + mid * 8) <= shared_key(larges + mid * 8);
    lo = before ? mid + 1 : lo;
    hi = before ? hi : mid;
  }
  const u32 end = A + S * 8;
  u32 ps = A + lo * 8, pl = larges + lo * 8 - 8;  // the heads of the two lists
  double sk = shared_key(ps), lk = shared_key(pl);
  u32 sp = shared_pos(ps), lp = shared_pos(pl);
#pragma unroll 4
  for (u32 k = k0; k < k1; ++k) {
    asm volatile(
        "{\n\t.reg .pred take, more, whole;\n\t.reg .f64 was, key, mass;\n\t.reg .b32 p, at, lo, hi, pos, alias;\n\t"
        ".reg .f32 prob;\n\t"
        "setp.ne.u32 more, %4, %6;\n\t"
        "setp.le.and.f64 take, %0, %1, more;\n\t"
        "selp.f64 was, %0, %1, take;\n\t"
        "selp.b32 p, %2, %3, take;\n\t"
        "@take add.u32 %4, %4, 8;\n\t"
        "@!take sub.u32 %5, %5, 8;\n\t"
        "selp.b32 at, %4, %5, take;\n\t"
        "ld.shared.v2.b32 {lo, hi}, [at];\n\t"
        "shr.u32 pos, hi, 20;\n\t"
        "lop3.b32 hi, hi, 0xFFFFF, 0x43300000, 0xEA;\n\t"
        "mov.b64 key, {lo, hi};\n\t"
        "@take mov.f64 %0, key;\n\t"
        "@take mov.b32 %2, pos;\n\t"
        "@!take mov.f64 %1, key;\n\t"
        "@!take mov.b32 %3, pos;\n\t"
        "sub.rn.f64 mass, was, %0;\n\t"
        "fma.rn.f64 mass, mass, 0d3D70000000000000, 0d3FF0000000000000;\n\t"  // in buckets (2^-40), exact
        "setp.ge.f64 whole, mass, 0d3FF0000000000000;\n\t"
        "selp.b32 alias, p, %3, whole;\n\t"
        "cvt.rn.f32.f64 prob, mass;\n\t"
        "mov.b32 lo, prob;\n\t"
        "mad.lo.u32 at, p, 8, %7;\n\t"
        "st.shared.v2.b32 [at], {lo, alias};\n\t}"
        : "+d"(sk), "+d"(lk), "+r"(sp), "+r"(lp), "+r"(ps), "+r"(pl)
        : "r"(end), "r"(out)
        : "memory");
  }
  if (k1 == n && (ps != end || pl != end)) dev_fail(err, DEV_ERR_INTERNAL, v, k0, 8);  // both lists are used up
}

// A: n + 1 words of shared memory; out: room for n slots there (and n / 2 more words at most, see below).
template <class Coop, int EPT>
__device__ __forceinline__ void build_list_f64(const Coop& co, u32 v, u32 off, u32 n, const float* __restrict__ w,
                                               Slot* __restrict__ slots, uint8_t* __restrict__ valid, uint2* A, uint2* out, u32* err) {
  constexpr int NT = Coop::NT;
  // Loops over a thread's weights are unrolled in steps of CH and left once `ept` of them are done (the same in all
  // threads); entries past the list's end have weight 0 and are taken out of the sums after the loop.
  constexpr int CH = 2;
  const u32 t = co.t;
  const u32 ept = (n + NT - 1) / NT;
  const u32 p0 = min(t * ept, n), cnt = min(ept, n - p0);
  const u32 over = min((ept + CH - 1) / CH * CH, (u32)EPT) - cnt;
#define SKW_EACH(k)                          \
  _Pragma("unroll") for (int b_ = 0; b_ < EPT; b_ += CH) { \
    if ((u32)b_ >= ept) break;               \
    _Pragma("unroll") for (int k = b_; k < b_ + CH; ++k)
#define SKW_EACH_END }
  // weights as integers: for positive floats the order of the bits is the order of the values, and what is
  // negative (or minus zero) becomes zero.  All loads are issued before any is used, so no loop exits among them.
  int wb[EPT];
  int top = 0;
  if constexpr (NT >= 8) {
    // Read in order across the threads and handed over through shared memory: read where they are needed, the
    // weights of a warp would lie in as many sectors as it has lanes.  An even number a thread is spread by one
    // word a thread, so that the threads start in different banks.
    int* stage = reinterpret_cast<int*>(out);
    const u32 per = ept & 1 ? 0u : 0xFFFFFFFFu / ept + 1;  // i / ept as a multiplication (i < 4096)
#pragma unroll
    for (int k = 0; k < EPT; ++k) wb[k] = t + k * NT < n ? __float_as_int(__ldg(w + t + k * NT)) : 0;
    SKW_EACH(k) {
      const u32 i = t + k * NT;
      if (i < n) stage[i + __umulhi(i, per)] = wb[k];
    }
    SKW_EACH_END
    co.sync();
    stage += t * (ept | 1);
#pragma unroll
    for (int k = 0; k < EPT; ++k) wb[k] = (u32)k < cnt ? stage[k] : 0;
  } else {
#pragma unroll
    for (int k = 0; k < EPT; ++k) wb[k] = (u32)k < cnt ? __float_as_int(__ldg(w + p0 + k)) : 0;
  }
  SKW_EACH(k) {
    wb[k] = max(wb[k], 0);
    top = max(top, wb[k]);
  }
  SKW_EACH_END
  top = co.template max<0>(top);
  if (top >= 0x7F800000) {  // infinities and NaNs count as zero
    top = 0;
    SKW_EACH(k) {
      if (wb[k] >= 0x7F800000) wb[k] = 0;
      top = max(top, wb[k]);
    }
    SKW_EACH_END
    top = co.template max<1>(top);
  }
  if (top == 0) {
    for (u32 p = t; p < n; p += NT) slots[(u64)off + p] = Slot{-1.0f, p};
    if (t == 0) valid[v] = 0;
    return;
  }
  if (top < (40 << 23)) {  // largest weight below 2^-87: scaled up (exactly) so that zeros and denormals quantise to 0
    SKW_EACH(k) { wb[k] = __float_as_int(__int_as_float(wb[k]) * 18446744073709551616.0f); }
    SKW_EACH_END
    top = __float_as_int(__int_as_float(top) * 18446744073709551616.0f);
  }
  const u64 shift = (u64)(1062 - (top >> 23)) << 52;  // exponent 896 + 39 - e
  double c[EPT];
  double Q = 0.0, W;
  SKW_EACH(k) {
    const double x = __longlong_as_double((long long)((u64)(u32)wb[k] * (1u << 29) + shift));
    c[k] = __dsub_rn(__dadd_rz(x, kTwo52), kTwo52);
    Q = __dadd_rn(Q, c[k]);
  }
  SKW_EACH_END
  co.scan(Q, W);
  const double all = __dmul_rn((double)n, kBucket);
  const double K = __ddiv_rn(all, W);
  const double all_b = __dadd_rn(all, kTwo52);
  auto mass_before = [&](double q) { return q == W ? all_b : __dadd_rz(__dmul_rn(q, K), kTwo52); };
  double g = mass_before(Q), D = 0.0, tD;
  u32 s = 0, S;
  double X = __dsub_rn(g, __dmul_rn((double)p0, kBucket));  // excess minus deficit before this thread
  SKW_EACH(k) {
    Q = __dadd_rn(Q, c[k]);
    const double gn = mass_before(Q);
    c[k] = __dsub_rn(kBucket, __dsub_rn(gn, g));  // what a small lacks, minus what a large has too much
    g = gn;
    count_small(c[k], D, s);
  }
  SKW_EACH_END
  D = __dsub_rn(D, __dmul_rn((double)over, kBucket));
  s -= over;
  co.scan(D, s, tD, S);
  X = __dadd_rn(X, D);
  D = __dadd_rn(D, kTwo52);
  const u32 at = (u32)__cvta_generic_to_shared(A);
  u32 ps = at + s * 8, pl = at + (n - (p0 - s)) * 8;
  const u32 tag = (p0 << 20) - kBiasHi;
  SKW_EACH(k) { put_entry(c[k], k, cnt, tag, D, X, ps, pl); }
  SKW_EACH_END
#undef SKW_EACH
#undef SKW_EACH_END
  if (t == 0) A[S] = list_entry(__dadd_rn(tD, kTwo52), 0);
  co.sync();
  if (S >= n) {  // mass conservation guarantees a large
    if (t == 0) dev_fail(err, DEV_ERR_INTERNAL, v, S, 7);
    for (u32 p = t; p < n; p += NT) slots[(u64)off + p] = Slot{1.0f, p};
  } else {
    const u32 to = (u32)__cvta_generic_to_shared(out);
    merge_f64<NT>(t, n, S, at, to, v, err);
    co.sync();
    for (u32 p = t; p < n; p += NT) reinterpret_cast<uint2*>(slots)[(u64)off + p] = out[p];
  }
  if (t == 0) valid[v] = 1;
}

}  // namespace skw

// Sliced complex GEMMs on tcgen05 for the P0 and Sigma stages.
//
// Why: a TF32/BF16 split with FP32 accumulation carries about 24 bits, and the
// GW contractions sum many terms of both signs, so their error stays near
// 1e-6 relative -- far from 1e-7 Ha absolute on Sigma.  Here each operand row
// is held, per round of at most 32 complex K, as three FP16 slices of its value
// relative to the row's exponent E (|x| < 2^E) (the Ozaki scheme: Ozaki, Ogita,
// Oishi, Rump, Numer. Algor. 59 (2012) 95-118; Mukunoki, Ozaki, Ogita, Imamura,
// ISC 2020 for FP16 tensor cores):
//   x 2^(15-E) = s0 + s1 + s2,  s0 a multiple of 2^6 (|s0| <= 2^15),
//   s1 a multiple of 2^(5-b) (|s1| <= 2^5), s2 the rest rounded to FP16,
// b = 9 bits for rounds of 3 or 4 octets of K, 10 for 2, 11 for 1.  What is
// left out is below 1.13 x 2^(E-32) and 2^(E-33) rms (s2 floats).  The products
// (i, j) with i + j <= 3 (8 MMAs per K step) go to four TMEM accumulators:
//   (0, 0): multiples of 2^12, at most 2^30 each: a round of 64 real terms stays
//           within 24 bits, so FP32 accumulation is exact;
//   (0, 1) and (1, 0), one each: 9 + b bits per term and the round's 6, 5 or 4: exact;
//   the rest: weight 2^-19 and less; its FP32 rounding lies near 2^-41.
// Dropped: s2 t2, below 2^-37 of the row-by-column scale.
//
// The FP64 contractions are the same chains with six slices: x 2^(8-E) = sum_p
// d_p 2^(-9p), |d_p| <= 2^8, d_0 .. d_4 integers and d_5 the rest rounded to FP16,
// so a row is held to about 2^(E-57) (FP64 itself holds each element to 2^-53 of
// itself: elements more than 2^4 below their row's largest have fewer bits here).
// The products of class i + j <= 6 (26 MMAs per K step) go to one
// accumulator per class; classes 0 to 3 are exact in FP32 (at most 4 products of
// 2^16 over 64 real terms), classes 4 to 6 have weight 2^-36 and less, class 7 is
// dropped (2^-61).  The drain sums the classes without error into three FP32
// numbers.  Against extended precision the error of P0 and Sigma (2-norm) is 0.6 to
// 1.8e-16, the FMA kernels' 1.0 to 5.2e-16; element by element (s+p+d, hexagonal and
// Gaussian-orbital crystals) the median is 0.5 to 1.9e-16 against 0.7 to 14e-16, the
// largest 0.2 to 9e-15 against 0.6 to 210e-15.  Their rate is the FP64 pipe's (2 FMA per cycle and SM); one
// complex output of K = 32 takes 64 cycles there and about 3 here.  Complex products use
// the real embedding A = [Ar Ai] (K interleaved), B rows (n, 0) = [Br -Bi],
// (n, 1) = [Bi Br], so D[r][(n,0)] = Re, D[r][(n,1)] = Im of sum_k A[r][k] B[n][k].
#include "kernels_oz.h"

#include <algorithm>
#include <cuda_fp16.h>

#include "tc_common.cuh"

namespace gwgb {

namespace {

constexpr int OZ_EMIN = -100, OZ_EMAX = 128;
// NS = 6: exponents of the images; a row without a nonzero value has -OZ_ELIM
constexpr int OZ_ELIM = 4000, OZ_ENONE = -1000000;

// E with |x| < 2^E for every |x| <= m (m >= 0), clamped to [OZ_EMIN, OZ_EMAX].
__device__ __forceinline__ int oz_exponent(float m) {
  const int e = (int)((__float_as_uint(m) >> 23) & 0xff) - 126;  // m = f 2^e, f in [0.5, 1)
  if (!(m > 0.f) || e < OZ_EMIN) return OZ_EMIN;
  return e > OZ_EMAX ? OZ_EMAX : e;
}

// 2^e for e in [-126, 127].
__device__ __forceinline__ float oz_pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// Two FP32 numbers per instruction (the drains are bound by their issue slots).
struct F2 {
  float x, y;
};
__device__ __forceinline__ F2 both(float a) { return {a, a}; }
#define OZ_F2_OP(op, ...)                                                                                   \
  F2 r;                                                                                                     \
  asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\n" op "mov.b64 {%0, %1}, c;\n}\n" \
      : "=f"(r.x), "=f"(r.y)                                                                                \
      : __VA_ARGS__);                                                                                       \
  return r
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  OZ_F2_OP("add.rn.f32x2 c, a, b;\n", "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  OZ_F2_OP("mul.rn.f32x2 c, a, b;\n", "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 d) {
  OZ_F2_OP(".reg .b64 d;\nmov.b64 d, {%6, %7};\nfma.rn.f32x2 c, a, b, d;\n", "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y),
           "f"(d.x), "f"(d.y));
}
#undef OZ_F2_OP
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, both(-1.f), a); }

// s = fl(a + b), e = a + b - s.
__device__ __forceinline__ void two_sum(F2 a, F2 b, F2 &s, F2 &e) {
  s = add2(a, b);
  const F2 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

// The three slices of h + l (v = fl(h + l), f = 2^(15-E)); adding and subtracting 1.5 2^(23+g) rounds
// to multiples of 2^g, and h f - s0 is exact.
__device__ __forceinline__ void oz_slice(F2 h, F2 l, F2 v, F2 f, F2 m1, F2 (&s)[3]) {
  constexpr float M0 = 1.5f * 536870912.f;  // 1.5 2^29
  const F2 r = fma2(v, f, both(M0));
  s[0] = add2(r, both(-M0));
  const F2 t = fma2(l, f, fma2(h, f, sub2(both(M0), r)));
  s[1] = sub2(add2(t, m1), m1);
  s[2] = sub2(t, s[1]);
}

// Unevaluated sums of three FP32 numbers; normalised: h the rounded value, m that of the rest.
struct Tri {
  F2 h, m, l;
};

// The value of the class sums D0 .. D3 and d4 = D4 + 2^-9 D5 + 2^-18 D6 (weights 2^(-9c)).  Carries instead of
// two-sums (26 steps against 44).  D0 to D3 are exact integers, sums of 64 (c + 1) products of digits; D2 and below leave
// room for a carry.  D3 with its carry stays within 2^24: a digit of 256 turns the sign of the next one (the remainder
// is at most half a unit), so a term whose four products of class 3 all have 256 in both factors and one sign has
// three of the other sign in class 4; a factor below 256 takes at least 1/256 of a product off class 3, twice what a
// whole product of class 4 carries.  In the worst mixture, three such products and one of 255 x 256, class 3 lacks 2/512 of a
// product and class 4 adds 1/512.  So each step is exact, but for the last bits of D4 to D6, which the tensor core
// rounds to 24 bits.  (The fourth digit of a drain's image may reach 260; class 3 could pass 2^24 only in rounds all of
// whose elements have the magnitude 2^E 512/513 to eight digits, and would lose its last bit there.)  NORM: normalised.
template <bool NORM> __device__ __forceinline__ Tri tri_of(const F2 (&d)[4], F2 d4) {
  const F2 W = both(0x1p-9f), MG = both(1.5f * 8388608.f), NM = both(-1.5f * 8388608.f), NB = both(-512.f);
  auto carry = [&](F2 x) { return add2(fma2(x, W, MG), NM); };  // x / 512 to an integer
  const F2 c4 = carry(d4);
  const F2 d3 = add2(d[3], c4), c3 = carry(d3);
  const F2 d2 = add2(d[2], c3), c2 = carry(d2);
  const F2 d1 = add2(d[1], c2), c1 = carry(d1);
  // a an integer, m a multiple of 2^-18 below 0.51, l below 2^-18 0.51: each zero or larger than the next
  const F2 a = add2(d[0], c1);
  const F2 m = fma2(fma2(c1, NB, d1), both(0x1p-9f), mul2(fma2(c2, NB, d2), both(0x1p-18f)));
  const F2 l = fma2(fma2(c3, NB, d3), both(0x1p-27f), mul2(fma2(c4, NB, d4), both(0x1p-36f)));
  if constexpr (!NORM) return {a, m, l};
  const F2 m1 = add2(m, l);
  Tri t;
  t.h = add2(a, m1);
  t.m = sub2(m1, sub2(t.h, a));
  t.l = sub2(l, sub2(m1, m));
  return t;
}

// a += b without normalising: sums and their errors stay in order of size, which leaves up to 4096 rounds within 2^-57
// of the largest partial sum (measured with a model of these steps; an FP64 addition rounds to 2^-53).  21 steps a
// round; normalised every time it was 36, and the FP32 pipe bounds the drains.
__device__ __forceinline__ void tri_add(Tri &a, const Tri &b) {
  F2 e1, m, e2, e3;
  two_sum(a.h, b.h, a.h, e1);
  two_sum(a.m, b.m, m, e2);
  two_sum(m, e1, a.m, e3);
  a.l = add2(add2(a.l, b.l), add2(e2, e3));
}

__device__ __forceinline__ void tri_norm(F2 &h, F2 &m, F2 &l) {
  two_sum(h, m, h, m);
  two_sum(m, l, m, l);
  two_sum(h, m, h, m);
}

// a + b for a zero or |a| > |b|: s the rounded sum, b what it leaves.
__device__ __forceinline__ F2 fast_two_sum(F2 a, F2 &b) {
  const F2 s = add2(a, b);
  b = sub2(b, sub2(s, a));
  return s;
}

// The six digits of h + m + l (nf = -2^(8-E)).  Of the negative: rounding by 1.5 2^23 - (1.5 2^23 + t) gives the digit of
// the positive number and, added, the remainder, three steps a digit.  Remainders are multiples of an ulp of the
// number they are left of and so zero or larger than the part that follows.
__device__ __forceinline__ void tri_digits(const Tri &x, F2 nf, F2 (&s)[6]) {
  const F2 MG = both(1.5f * 8388608.f), B = both(512.f);
  auto digit = [&](F2 a, F2 f, F2 &d) {  // a f = -d + what is returned
    d = sub2(MG, fma2(a, f, MG));
    return fma2(a, f, d);
  };
  F2 t = digit(x.h, nf, s[0]), te = mul2(x.m, nf);
  t = fast_two_sum(t, te);
  te = fma2(x.l, nf, te);
  t = digit(t, B, s[1]);
  t = digit(t, B, s[2]);
  te = mul2(te, both(262144.f));
  t = fast_two_sum(t, te);
  t = digit(t, B, s[3]);
  t = digit(t, B, s[4]);
  s[5] = fma2(te, both(-134217728.f), mul2(t, both(-512.f)));  // te 2^27
}

// 2^e for any e, 0 below the FP32 range.
__device__ __forceinline__ float oz_pow2c(int e) { return e < -126 ? 0.f : oz_pow2(min(e, 127)); }

// The rounding constant of s1 for an image of nks octets of K.
__device__ __forceinline__ float oz_m1(int nks) {
  return nks == 1 ? 1.5f * 131072.f : nks == 2 ? 1.5f * 262144.f : 1.5f * 524288.f;  // 1.5 2^(28-b)
}

__device__ __forceinline__ uint32_t h2(F2 a) {
  const __half2 v = __floats2half2_rn(a.x, a.y);
  return *reinterpret_cast<const uint32_t *>(&v);
}

// One 32-byte sector (an octet of one row and plane), its 16-byte halves
// swapped in rows 4-7 of every 8 (the 32-byte swizzle).
__device__ __forceinline__ void st_octet(char *p, const uint32_t (&w)[8], bool swap) {
  uint32_t v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = swap ? w[j ^ 4] : w[j];
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// K-major operand in the 32-byte swizzle: rows of 32 bytes, 8-row groups 256 bytes apart.
__device__ __forceinline__ uint64_t sw32_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;            // leading dimension: unused, K is one atom wide
  d |= (uint64_t)(256 >> 4) << 32;   // stride between 8-row groups
  d |= (uint64_t)1 << 46;            // descriptor version of the sm_100 family
  d |= (uint64_t)6 << 61;            // SWIZZLE_32B
  return d;
}
// D = F32, A = B = F16, both K-major.
__device__ __forceinline__ uint32_t idesc_f16(int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);
}

// 32 lanes x 8 consecutive 32-bit columns; the caller waits (tmem_wait_ld) before use.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void bulk_load(uint32_t dst, const char *src, uint32_t bytes, uint64_t *mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(tc::smem_u32(mbar))
               : "memory");
}
__device__ __forceinline__ void expect_tx(uint64_t *mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(mbar)), "r"(bytes)
               : "memory");
}

// The sequence of rounds of one task: `outer` row tiles of R rounds (stages 1
// and 2, the column operand held over the row tiles), or R rounds (stage 3).
template <int NS, int STAGE> struct Job {
  static constexpr int OCT = OzCfg<NS>::OCT;
  int outer, R, noct, kos;
  int G;                 // row tiles per accumulator set
  const char *a, *b;
  int64_t atile;
  const OzRnd *rt;
  __device__ __forceinline__ void init(const OzArgs &g, const OzTask &t) {
    rt = nullptr;
    if constexpr (STAGE == 0) {
      const OzS1 d = static_cast<const OzS1 *>(g.desc)[t.d];
      const OzCol1 c = static_cast<const OzCol1 *>(g.aux1)[t.i];
      kos = d.kos;
      R = (kos + OCT - 1) / OCT;
      outer = t.n;
      noct = c.ngrp * c.gs;
      atile = (int64_t)NS * kos * 4096 + 512 * R;
      a = g.A + d.a + t.m0 * atile;
      b = g.B + c.b;
    } else if constexpr (STAGE == 1) {
      const OzS2 d = static_cast<const OzS2 *>(g.desc)[t.d];
      const int tau = t.i & 0xffff, zt = t.i >> 16;
      kos = d.kos;
      R = (kos + OCT - 1) / OCT;
      outer = t.n;
      noct = min(OCT, d.zos - zt * OCT);
      atile = d.t2bytes;
      a = g.A + d.a + ((int64_t)tau * d.nt2 + t.m0) * atile;
      b = g.B + d.b + tau * d.bt + zt * d.bz;
    } else {
      const OzS3 d = static_cast<const OzS3 *>(g.desc)[t.d];
      const int f = t.i & 0xffff, ct = t.i >> 16;
      kos = 0;
      R = d.nkr;
      outer = t.n;
      noct = min(d.oct, (d.N + 7) / 8 - ct * d.oct);
      atile = d.fbytes;
      a = g.A + d.a + f * d.fbytes;
      b = g.B + d.b + ct * d.bz;
      rt = static_cast<const OzRnd *>(g.aux1) + d.rt;
    }
    G = STAGE == 0 ? 1 : OCT / noct;
  }
  // Round r (stage 3: from the round table, read one round ahead).
  __device__ __forceinline__ OzRnd round(int r) const {
    if constexpr (STAGE == 2) return rt[min(r, R - 1)];
    return {0, 0, min(OCT, kos - r * OCT), 0};
  }
  __device__ __forceinline__ const char *aptr(int m, int r, const OzRnd &q) const {
    return a + m * atile + (STAGE == 2 ? (int64_t)q.a16 * 16 : r * oz_abytes(NS, OCT));
  }
  __device__ __forceinline__ const char *bptr(int r, const OzRnd &q) const {
    return b + noct * (STAGE == 2 ? (int64_t)q.b16 * 16 : r * oz_bbytes1(NS, OCT));
  }
};

constexpr int OZ_RING = 8;              // largest operand ring of a set
constexpr int OZ_SC = 16;               // scale rings of a set: deeper than its operand ring plus its row tiles
constexpr int OZ_SMEM = 200 * 1024;
// Drain warps (then per accumulator set one that copies and one that issues the MMAs): three slices take two
// octets per thread in 8 warps (stage 1 of Sigma, hexagonal 8 k, 7.5 ms against 8.8 with one octet in 16 warps),
// six slices one octet in 16 warps (s+p+d: 24 ms an iteration against 33 when that was measured: unrolled over two
// octets the code misses the instruction cache).
template <int NS> constexpr int oz_drain = 4 * OzCfg<NS>::OCT / OzCfg<NS>::HO;
template <int NS> constexpr int oz_threads = NS == 6 ? 640 : 32 * (oz_drain<NS> + 2 * OzCfg<NS>::SETS);

// One lane of a converged warp.  The copy and MMA loops are warp-uniform and
// elect a lane only around the instruction itself: their descriptors then stay in
// uniform registers.  In a one-lane branch every MMA took 161 cycles to issue,
// whatever its N; this way the N = 64 MMA takes 48, its operand reads.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred P;\nelect.sync _|P, 0xffffffff;\nselp.b32 %0, 1, 0, P;\n}\n" : "=r"(p));
  return p != 0;
}

// Ring position.
struct Ring {
  int slot = 0, phase = 0, n;
  __device__ __forceinline__ explicit Ring(int n_) : n(n_) {}
  __device__ __forceinline__ void next() {
    if (++slot == n) {
      slot = 0;
      phase ^= 1;
    }
  }
};

// The MMAs of one K step, classes C0 to C1 of slice products (one lane).  NS = 3: accumulators (0,0) | (0,1) |
// (1,0) | the rest; NS = 6: one per class.
template <int NS, int C0, int C1>
__device__ __forceinline__ void oz_mmas(uint32_t d0, uint32_t a0, uint32_t b0, uint32_t bstep, uint32_t id,
                                        uint32_t more) {
  constexpr int NR = 16 * OzCfg<NS>::OCT;
#pragma unroll
  for (int c = C0; c <= C1; ++c)
#pragma unroll
    for (int p = 0; p < NS; ++p) {
      const int q = c - p;
      if (q < 0 || q >= NS) continue;
      const int acc = NS == 6 ? c : c == 0 ? 0 : c == 1 ? 1 + p : 3;
      const bool fresh = NS == 6 ? p == max(0, c - NS + 1) : c < 2 || (c == 2 && p == 0);
      tc::mma_bf16(d0 + acc * NR, sw32_desc(a0 + p * 4096u), sw32_desc(b0 + q * bstep), id,
                   fresh ? more : 1u);  // kind::f16, types from the descriptor
    }
}

// Persistent warp-specialised GEMM over operand images.  Bound, three slices: HBM in
// stages 2 and 3 (hexagonal 8 k, Sigma: 6.1 and 5.6 TB/s of 6.8), the drains in stage 1
// (2500 cycles per accumulator set, its MMAs 880); six slices: the drains' FP32 work, in
// stage 3 about as long as the MMAs.  The operands need no CUDA-core work at all, a K step
// (8 complex) is 8 or 26 MMAs, and the two accumulator sets of three slices let
// one round multiply while the other drains.  Operands stream through rings of
// segments of SEG K steps; stages 1 and 2 hold the column operand of a task over
// its row tiles.  The issue of an MMA blocks its warp while the tensor pipe is
// busy, so whatever that warp does in between (barriers, commits, the round
// table) adds to the time: measured, 200 idle cycles per 4 K steps cost 240.  Each
// accumulator set therefore has a copy and an MMA warp and rings of its own, and
// one set's loop overhead is hidden behind the other's MMAs (two issuing warps:
// 1200 idle cycles cost 100).  Stage 3 of the hexagonal 8 k crystal (three
// slices), Sigma: one K step per segment and one MMA warp 10.4 ms, segments of four
// 6.5; an MMA warp per set, with segments of two in rings of its own, 6.2.
// Six slices have room for one set in TMEM.  There a round's MMAs go in two groups, the
// classes 4 to 6 (16 of the 26 products of a K step) and 0 to 3, with barriers of their
// own: the drain reads the high classes while the low ones multiply and the low ones
// while the next round's high ones do.  In one group the multiplies and the TMEM reads
// of a set took turns: stage 3 of Sigma, hexagonal 4 k, 5.33 ms, in two 4.45.
// A column tile of one octet (two) fills a quarter (half) of an accumulator set, so
// stages 2 and 3 put G = OCT / noct row tiles into one.
//
// Every wait is bounded: a wait that runs out sets the error word and an abort
// flag; the copy and MMA roles then leave, the drain warps walk on through
// their work without waiting (their named barriers stay matched).  Copies and
// MMAs in flight are waited for (bounded) before TMEM is released.
// MULTI (stages 1 and 2): tasks with more than one round of K.
template <int NS, int STAGE, bool MULTI>
__global__ void __launch_bounds__(oz_threads<NS>, 1) oz_gemm_kernel(const OzArgs g) {
  constexpr int OCT = OzCfg<NS>::OCT, NACC = OzCfg<NS>::NACC, HO = OzCfg<NS>::HO, DW = oz_drain<NS>;
  constexpr int NR = 16 * OCT, SETC = NACC * NR;
  constexpr int SEG = STAGE == 2 ? OzCfg<NS>::SEG3 : OzCfg<NS>::SEG;
  constexpr uint32_t SA = NS * 4096, SB = NS * 512 * OCT;  // one K step
  constexpr int SETS = OzCfg<NS>::SETS;
  static_assert(SETS * SETC <= 512, "the accumulator sets must fit TMEM");
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t tslot;
  __shared__ __align__(8) uint64_t full[SETS][OZ_RING], emptyA[SETS][OZ_RING], emptyB[SETS][OZ_RING], fullB[2],
      done[SETS], tfree[SETS], doneH, tfreeH, last;
  __shared__ __align__(16) float sA[SETS][OZ_SC][OZ_M], sB[SETS][OZ_SC][8 * OCT];
  __shared__ float gmax[2][OCT / HO][OZ_M];  // exchange n of a warp in gmax[n & 1]
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (warp == 0) tc::tmem_alloc(&tslot, 512);
  if (tid == 0) {
    for (int j = 0; j < SETS; ++j) {
      for (int k = 0; k < OZ_RING; ++k) {
        tc::mbar_init(&full[j][k], 1);
        tc::mbar_init(&emptyA[j][k], 1);
        tc::mbar_init(&emptyB[j][k], STAGE == 2 ? 1 : SETS);  // stages 1 and 2 use emptyB[0]
      }
      tc::mbar_init(&done[j], 1);
      tc::mbar_init(&tfree[j], DW);
    }
    tc::mbar_init(&fullB[0], 1);
    tc::mbar_init(&fullB[1], 1);
    tc::mbar_init(&doneH, 1);
    tc::mbar_init(&tfreeH, DW);
    tc::mbar_init(&last, SETS);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tm = __shfl_sync(0xffffffffu, tslot, 0);
  // Bounded wait of a converged warp; false (in every lane) when it ran out (error word and abort
  // flag set) or another role aborted.  Each poll may suspend for up to 20 us (hint).
  auto poll = [&](uint64_t *b, uint32_t par) -> bool {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(tc::smem_u32(b)), "r"(par), "r"(20000u)
        : "memory");
    return ok != 0;
  };
  auto bwait = [&](uint64_t *b, uint32_t par) -> bool {
    if (__all_sync(0xffffffffu, poll(b, par))) return true;
    bool hit = false;
    for (int rep = 0; rep < 256 && !hit; ++rep) {
      for (int it = 0; it < 256 && !hit; ++it) hit = poll(b, par);
      if (!hit && *(volatile int *)&abort_flag) break;
      if (!hit && rep == 255) {
        atomicExch(g.err, 1);
        *(volatile int *)&abort_flag = 1;
      }
    }
    return __all_sync(0xffffffffu, hit);
  };
  // rings: nA segments of A per set, then nB segments of B per set (stage 3) or tasksB tasks' B of nB K steps
  const uint32_t smA0 = tc::smem_u32(smem), smB0 = smA0 + (uint32_t)(SETS * g.nA) * SEG * SA;

  // six slices: registers of the drain and other warps, 512 x 112 + 128 x 32 and 512 x 104 + 128 x 56 of the launch's
  // 640 x 96 (which of the two spills less; 150 bytes spilled in stage 2 took Sigma's, hexagonal 4 k, from 4.5 to 7.0 ms)
  constexpr int DREG = STAGE == 1 ? 104 : 112, OREG = STAGE == 1 ? 56 : 32;
  if (warp < DW) {
    if constexpr (NS == 6) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DREG));
    // ------------------------------ drain ------------------------------
    // warp w: TMEM lanes (rows) 32 (w & 3) .. + 31, octets HO (w >> 2) .. + HO - 1 of the set.
    // The rows' destinations are read while the set still multiplies.
    const int lq = warp & 3, os0 = HO * (warp >> 2), row = 32 * lq + lane;
    const uint32_t tbase = tm + ((uint32_t)(32 * lq) << 16) + 16u * os0;
    int n = 0, xch = 0, i0[SETS] = {}, j0[SETS] = {};  // fills, exchanges; row tiles and column images by set
    bool dead = false;
    OzTask tk1{};
    if (blockIdx.x < (unsigned)g.ntasks) tk1 = g.tasks[blockIdx.x];
    for (int ti = blockIdx.x; ti < g.ntasks; ti += gridDim.x) {
      const OzTask tk = tk1;
      if (ti + (int)gridDim.x < g.ntasks) tk1 = g.tasks[ti + gridDim.x];
      Job<NS, STAGE> job;
      job.init(g, tk);
      // row tile in the set, octet in the tile, valid columns of the octet
      int gi[HO], oct[HO], nv[HO];
#pragma unroll
      for (int q = 0; q < HO; ++q) {
        gi[q] = (os0 + q) / job.noct;
        oct[q] = os0 + q - gi[q] * job.noct;
      }
      // stage 1: the row and its destination
      int rg = 0, M = 0, nL = 1, tau = 0, Lr = 0, dtau = 0, dL = 0, gs = 1, glog = 0, nt2 = 1, nLp = 0, nx = 0;
      int slot0 = 0, ksq[HO], xq[HO];  // first slot; K step and x of the octets
      int64_t t2bytes = 0;
      char *xbase = g.X;
      // stage 2
      const OzRow *rows = nullptr;
      OzRow rw[HO];
      if constexpr (STAGE == 0) {
        const OzS1 d = static_cast<const OzS1 *>(g.desc)[tk.d];
        const OzCol1 col = static_cast<const OzCol1 *>(g.aux1)[tk.i];
        const OzDst1 d1 = static_cast<const OzDst1 *>(g.aux2)[col.dst];
        M = d.M;
        nL = d.nL;
        gs = col.gs;
        slot0 = d1.slot0;
        nLp = d1.nLp;
        nx = d1.nx;
        nt2 = d1.nt2;
        t2bytes = d1.t2bytes;
        xbase += d1.base + col.yoff;
        rg = tk.m0 * OZ_M + row;
        tau = rg / nL;
        Lr = rg - tau * nL;
        dtau = OZ_M / nL;
        dL = OZ_M - dtau * nL;
#pragma unroll
        for (int q = 0; q < HO; ++q) {
          const int grp = oct[q] / gs;
          ksq[q] = oct[q] - grp * gs;
          xq[q] = col.x0 + grp;
          nv[q] = col.ny - 8 * ksq[q];
                  }
      } else if constexpr (STAGE == 1) {
        const OzS2 d = static_cast<const OzS2 *>(g.desc)[tk.d];
        gs = job.noct;
        glog = d.glog;
        tau = tk.i & 0xffff;
        xbase += (tk.i >> 16) * oz_abytes(NS, OCT);
        rows = static_cast<const OzRow *>(g.aux1) + d.rows + tk.m0 * OZ_M + row;
#pragma unroll
        for (int q = 0; q < HO; ++q) {
          nv[q] = d.nz - 8 * ((tk.i >> 16) * OCT + oct[q]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < HO; ++q) {
          const OzS3 &d = static_cast<const OzS3 *>(g.desc)[tk.d];
          nv[q] = d.N - 8 * ((tk.i >> 16) * d.oct + oct[q]);
        }
      }
      for (int m0 = 0; m0 < job.outer; m0 += job.G) {
        const int Gm = min(job.G, job.outer - m0);
        if constexpr (STAGE == 1) {  // used after the wait for the accumulators
#pragma unroll
          for (int q = 0; q < HO; ++q) {
            rw[q].pk = OZ_NOROW;
            if (gi[q] < Gm) rw[q] = rows[(m0 + gi[q]) * OZ_M];
          }
        }
        // this thread's octets: value H + L (NS = 3), (H + M + L) 2^ex (NS = 6)
        F2 H[HO][8], L[HO][8], M3[NS == 6 ? HO : 1][8];
        int ex[HO];
#pragma unroll
        for (int q = 0; q < HO; ++q) {
          ex[q] = 0;
#pragma unroll
          for (int e = 0; e < 8; ++e) H[q][e] = L[q][e] = M3[NS == 6 ? q : 0][e] = both(0.f);
        }
        for (int r = 0; r < job.R; ++r, ++n) {
          const int set = n % SETS, ia = set ? i0[SETS - 1] : i0[0], jb = STAGE != 2 ? j0[0] + r : set ? j0[SETS - 1] : j0[0];
          (set ? i0[SETS - 1] : i0[0]) += Gm;
          if (STAGE == 2) ++(set ? j0[SETS - 1] : j0[0]);
          F2 d4[NS == 6 ? 8 : 1];  // six slices: classes 4 to 6 of this octet (HO is 1)
          if constexpr (NS == 6) {
            if (!dead) dead = !bwait(&doneH, n & 1);
            if (dead) continue;
            tc::fence_after_sync();
            if (gi[0] < Gm) {
              const F2 W = both(0x1p-9f);
#pragma unroll
              for (int hf = 0; hf < 4; ++hf) {
                if (2 * hf >= nv[0]) continue;
                uint32_t x[3][4];
#pragma unroll
                for (int c = 0; c < 3; ++c) tmem_ld4(tbase + (4 + c) * NR + 4 * hf, x[c]);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  auto at = [&](int c) { return F2{__uint_as_float(x[c][2 * e]), __uint_as_float(x[c][2 * e + 1])}; };
                  d4[2 * hf + e] = fma2(fma2(at(2), W, at(1)), W, at(0));
                }
              }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&tfreeH);
          }
          if (!dead) dead = !bwait(&done[set], (n / SETS) & 1);
          if (dead) continue;
          tc::fence_after_sync();
          const bool first = STAGE == 2 || MULTI ? r == 0 : true;
#pragma unroll
          for (int q = 0; q < HO; ++q) {
            if (gi[q] >= Gm) continue;
            const float *sbp = sB[STAGE == 2 ? set : 0][jb & (OZ_SC - 1)] + 8 * oct[q];
            const uint32_t base = tbase + (uint32_t)(set * SETC) + 16u * q;
            const float sa = sA[set][(ia + gi[q]) & (OZ_SC - 1)][row];
            if constexpr (NS == 3) {
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                if (4 * hf >= nv[q]) continue;
                uint32_t x0[8], x1[8], x2[8], x3[8];
                tmem_ld8(base + 8 * hf, x0);
                tmem_ld8(base + NR + 8 * hf, x1);
                tmem_ld8(base + 2 * NR + 8 * hf, x2);
                tmem_ld8(base + 3 * NR + 8 * hf, x3);
                const float4 sb4 = *reinterpret_cast<const float4 *>(sbp + 4 * hf);
                const float sb[4] = {sb4.x, sb4.y, sb4.z, sb4.w};
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  auto at = [&](const uint32_t(&x)[8]) {
                    return F2{__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1])};
                  };
                  const int c = 4 * hf + e;
                  const F2 sc = both(sa * sb[e]);
                  const F2 lo = add2(add2(at(x1), at(x2)), at(x3));
                  if (first) {
                    H[q][c] = mul2(at(x0), sc);
                    L[q][c] = mul2(lo, sc);
                  } else {
                    F2 s, er;
                    two_sum(H[q][c], mul2(at(x0), sc), s, er);
                    H[q][c] = s;
                    L[q][c] = add2(L[q][c], fma2(lo, sc, er));
                  }
                }
              }
            } else {
              // exponent of the row and of this octet's columns, relative column factors
              const int4 b0 = *reinterpret_cast<const int4 *>(sbp), b1 = *reinterpret_cast<const int4 *>(sbp + 4);
              const int eb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
              const int em = max(max(max(eb[0], eb[1]), max(eb[2], eb[3])), max(max(eb[4], eb[5]), max(eb[6], eb[7])));
              const int er = __float_as_int(sa) + em;
              float fo = 1.f, fn = 1.f;  // factors of the sum so far and of this round
              if (first) {
                ex[q] = er;
              } else if (er > ex[q]) {
                fo = oz_pow2c(ex[q] - er);
                ex[q] = er;
              } else {
                fn = oz_pow2c(er - ex[q]);
              }
#pragma unroll
              for (int hf = 0; hf < 4; ++hf) {
                if (2 * hf >= nv[q]) continue;
                uint32_t x[4][4];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld4(base + c * NR + 4 * hf, x[c]);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int i = 2 * hf + e;
                  F2 d[4];
#pragma unroll
                  for (int c = 0; c < 4; ++c) d[c] = {__uint_as_float(x[c][2 * e]), __uint_as_float(x[c][2 * e + 1])};
                  Tri t = tri_of<STAGE != 2 && !MULTI>(d, d4[i]);
                  const F2 sc = both(oz_pow2c(eb[i] - em) * fn);
                  t = {mul2(t.h, sc), mul2(t.m, sc), mul2(t.l, sc)};
                  if (!first) {
                    const F2 fo2 = both(fo);
                    Tri o{mul2(H[q][i], fo2), mul2(M3[q][i], fo2), mul2(L[q][i], fo2)};
                    tri_add(o, t);
                    t = o;
                  }
                  H[q][i] = t.h;
                  M3[q][i] = t.m;
                  L[q][i] = t.l;
                }
              }
            }
          }
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&tfree[set]);
        }
        if constexpr (NS == 6 && STAGE != 2 && MULTI) {
#pragma unroll
          for (int e = 0; e < 8; ++e) tri_norm(H[0][e], M3[0][e], L[0][e]);
        }
        if constexpr (STAGE == 2) {  // FP64 partial of this K slice
          const OzS3 d = static_cast<const OzS3 *>(g.desc)[tk.d];
#pragma unroll
          for (int q = 0; q < HO; ++q) {
            const int fr = ((tk.i & 0xffff) + m0 + gi[q]) * OZ_M + row, n0 = d.N - nv[q];
            if (gi[q] >= Gm || fr >= d.M || dead) continue;
            const int t = fr / d.nx, x = fr - t * d.nx;
            double2 *o = g.part + d.part + (int64_t)t * d.elems + (int64_t)x * d.sx;
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < nv[q]) {
                const F2 h = H[q][e], l = L[q][e];
                double re, im;
                if constexpr (NS == 6) {
                  const F2 m = M3[q][e];
                  re = scalbn((double)h.x + ((double)m.x + (double)l.x), ex[q]);
                  im = scalbn((double)h.y + ((double)m.y + (double)l.y), ex[q]);
                } else {
                  re = (double)h.x + (double)l.x;
                  im = (double)h.y + (double)l.y;
                }
                o[(int64_t)(n0 + e) * d.sn] = make_double2(re, im);
              }
          }
        } else {
          // largest component of each octet, as a value (NS = 3) or an exponent (NS = 6)
          bool valid[HO];
          float mx[HO];
          int ee[HO];
#pragma unroll
          for (int q = 0; q < HO; ++q) {
            valid[q] = gi[q] < Gm && (STAGE == 0 ? rg < M : rw[q].pk != OZ_NOROW);
            float mo[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const F2 v = NS == 3 ? add2(H[q][e], L[q][e]) : H[q][e];
              mo[e] = fmaxf(fabsf(v.x), fabsf(v.y));
            }
            mx[q] = fmaxf(fmaxf(fmaxf(mo[0], mo[1]), fmaxf(mo[2], mo[3])),
                          fmaxf(fmaxf(mo[4], mo[5]), fmaxf(mo[6], mo[7])));
            ee[q] = mx[q] > 0.f || mx[q] != mx[q] ? oz_exponent(mx[q]) + ex[q] : OZ_ENONE;
            if (!valid[q]) {
              mx[q] = 0.f;
              ee[q] = OZ_ENONE;
            }
          }
          // Octets that share an exponent: gs = 2 the pairs (0, 1) and (2, 3), gs > 2 all of them (octets past the
          // third are then invalid and do not count).  Beyond a thread's own they are in the other warps of its
          // lane quarter: gmax, one barrier per exchange.  The buffers alternate by exchange (gs is the same in these
          // warps), not by tile: a warp writes buffer n & 1 again in exchange n + 2, after the barrier of n + 1, which
          // every warp reaches only when it has read exchange n.  By tile, one without an exchange in between left
          // nothing to order the two (the warps of a quarter may be two fills of the accumulators apart).
          if constexpr (HO == 2) {
            if (gs >= 2) {
              mx[0] = fmaxf(mx[0], mx[1]);
              if (gs > 2) {
                gmax[xch & 1][os0 / HO][row] = mx[0];
                asm volatile("bar.sync %0, %1;" ::"r"(1 + lq), "n"(32 * OCT / HO) : "memory");
                mx[0] = fmaxf(mx[0], gmax[xch & 1][1 - os0 / HO][row]);
                ++xch;
              }
              mx[1] = mx[0];
            }
          } else if (gs > 1) {
            gmax[xch & 1][os0][row] = __int_as_float(ee[0]);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + lq), "n"(32 * OCT / HO) : "memory");
            if (gs == 2) {
              ee[0] = max(ee[0], __float_as_int(gmax[xch & 1][os0 ^ 1][row]));
            } else {
#pragma unroll
              for (int k = 0; k < OCT; ++k) ee[0] = max(ee[0], __float_as_int(gmax[xch & 1][k][row]));
            }
            ++xch;
          }
          if constexpr (STAGE == 1) {  // rows L of one K round share the exponent of their (tau, x)
            for (int dlt = 1; dlt < (1 << glog); dlt <<= 1) {
#pragma unroll
              for (int q = 0; q < HO; ++q) {
                if constexpr (NS == 6) {
                  ee[q] = max(ee[q], __shfl_xor_sync(0xffffffffu, ee[q], dlt));
                } else {
                  mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], dlt));
                }
              }
            }
          }
#pragma unroll
          for (int q = 0; q < HO; ++q) {
            if (!valid[q] || dead) continue;
            // the row's blob, its row and K step there
            char *blob = xbase;
            int nksb = gs, rr, ks;
            if constexpr (STAGE == 0) {
              const int Lq = Lr & ~3, slot = slot0 + Lq * nx + xq[q] * min(4, nLp - Lq) + (Lr & 3);
              blob += ((int64_t)tau * nt2 + (slot >> 7)) * t2bytes;
              rr = slot & 127;
              ks = ksq[q];
            } else {
              const uint32_t pk = rw[q].pk;
              const int fr = tau * (int)((pk >> 8) & 255) + (int)(pk & 255);
              if (glog) nksb = (int)(pk >> 24);
              ks = (int)((pk >> 16) & 255) + oct[q];
              blob += rw[q].base + (int64_t)(fr >> 7) * rw[q].f16 * 16;
              rr = fr & 127;
            }
            uint32_t w[NS][8];
            float scale;
            const int e2 = NS == 3 ? oz_exponent(mx[q]) : max(ee[q], -OZ_ELIM);
            if constexpr (NS == 3) {
              scale = oz_pow2(e2 - 15);
            } else {
              scale = __int_as_float(e2 - 8);
            }
            // NS = 6: -2^(8 - e2 + ex); e2 - ex is at least the exponent of an FP32 value
            const F2 f = both(NS == 3 ? oz_pow2(15 - e2) : -oz_pow2c(8 - e2 + ex[q])), m1 = both(oz_m1(nksb));
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              if (e == 4 && nv[q] <= 4) {  // the second half is padding
#pragma unroll
                for (int p = 0; p < NS; ++p) w[p][4] = w[p][5] = w[p][6] = w[p][7] = 0u;
                break;
              }
              F2 sl[NS];
              if constexpr (NS == 3)
                oz_slice(H[q][e], L[q][e], add2(H[q][e], L[q][e]), f, m1, sl);
              else
                tri_digits({H[q][e], M3[q][e], L[q][e]}, f, sl);
#pragma unroll
              for (int p = 0; p < NS; ++p) w[p][e] = h2(sl[p]);
            }
            char *o = blob + ks * (int)SA + rr * 32;
            const bool sw = (rr >> 2) & 1;
#pragma unroll
            for (int p = 0; p < NS; ++p) st_octet(o + p * 4096, w[p], sw);
            if (ks == 0) reinterpret_cast<float *>(blob + (int64_t)nksb * SA)[rr] = scale;
          }
        }
        if constexpr (STAGE == 0) {  // the next row tile
          rg += OZ_M;
          tau += dtau;
          Lr += dL;
          if (Lr >= nL) {
            Lr -= nL;
            ++tau;
          }
        }
      }
      if (STAGE != 2) j0[0] += job.R;
    }
  } else {
    if constexpr (NS == 6) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OREG));
    if (warp < DW + SETS) {
      // ------------------------------ copies ------------------------------
      const int set = warp - DW;
      const uint32_t smA = smA0 + set * (g.nA * SEG * SA), smB = smB0 + (STAGE == 2 ? set * (g.nB * SEG * SB) : 0);
      Ring ra(g.nA), rb(STAGE == 2 ? g.nB : g.tasksB);
      int ia = 0, ib = 0, na = 0, nb = 0, n = 0;  // segments (of A, of B or tasks), scales, fills of the sets
      bool ok = true;
      for (int ti = blockIdx.x; ti < g.ntasks && ok; ti += gridDim.x) {
        Job<NS, STAGE> job;
        job.init(g, g.tasks[ti]);
        const uint32_t bb = (uint32_t)(job.noct * NS * 512), sb = (uint32_t)(32 * job.noct);
        if (STAGE != 2 && set == 0) {  // the task's column operand, all rounds
          if (ib >= g.tasksB && !bwait(&emptyB[0][rb.slot], rb.phase ^ 1)) { ok = false; break; }
          if (elect_one()) {
            uint64_t *f = &fullB[rb.slot];
            expect_tx(f, job.kos * bb + job.R * sb);
            for (int r = 0; r < job.R; ++r) {
              const int nks = min(OCT, job.kos - r * OCT);
              const char *bp = job.bptr(r, OzRnd{});
              bulk_load(smB + rb.slot * (g.nB * SB) + r * OCT * bb, bp, nks * bb, f);
              bulk_load(tc::smem_u32(sB[0][(nb + r) & (OZ_SC - 1)]), bp + nks * bb, sb, f);
            }
          }
          __syncwarp();
          nb += job.R;
          rb.next();
          ++ib;
        }
        for (int m0 = 0; m0 < job.outer && ok; m0 += job.G) {
          const int Gm = min(job.G, job.outer - m0);
          int r = (n ^ set) & (SETS - 1);  // this set's rounds
          n += job.R;
          OzRnd nx = job.round(r);
          for (; r < job.R && ok; r += SETS) {
            const OzRnd q = nx;
            nx = job.round(r + SETS);
            for (int gi = 0; gi < Gm && ok; ++gi) {
              const bool withb = STAGE == 2 && gi == 0;
              const char *ap = job.aptr(m0 + gi, r, q), *bp = job.bptr(r, q);
              for (int ks = 0; ks < q.nks; ks += SEG) {
                const int nk = min(SEG, q.nks - ks);
                if (ia >= g.nA && !bwait(&emptyA[set][ra.slot], ra.phase ^ 1)) { ok = false; break; }
                if (withb && ib >= g.nB && !bwait(&emptyB[set][rb.slot], rb.phase ^ 1)) { ok = false; break; }
                if (elect_one()) {
                  uint64_t *f = &full[set][ra.slot];
                  expect_tx(f, nk * SA + (ks == 0 ? 512u : 0u) + (withb ? nk * bb + (ks == 0 ? sb : 0u) : 0u));
                  bulk_load(smA + ra.slot * (SEG * SA), ap + ks * SA, nk * SA, f);
                  if (withb) bulk_load(smB + rb.slot * (SEG * SB), bp + ks * bb, nk * bb, f);
                  if (ks == 0) {
                    bulk_load(tc::smem_u32(sA[set][na & (OZ_SC - 1)]), ap + q.nks * SA, 512, f);
                    if (withb) bulk_load(tc::smem_u32(sB[set][nb & (OZ_SC - 1)]), bp + q.nks * bb, sb, f);
                  }
                }
                __syncwarp();
                if (withb) {
                  rb.next();
                  ++ib;
                }
                ra.next();
                ++ia;
              }
              ++na;
              if (withb) ++nb;
            }
          }
        }
      }
      // every copy issued has landed before the CTA may end
      Ring rw(g.nA);
      const int first = max(0, ia - g.nA);
      for (int q = 0; q < ia; ++q) {
        if (q >= first) tc::mbar_wait(&full[set][rw.slot], rw.phase, 4000000);
        rw.next();
      }
      if (STAGE != 2 && set == 0) {
        Ring rv(g.tasksB);
        for (int q = 0; q < ib; ++q) {
          if (q >= ib - g.tasksB) tc::mbar_wait(&fullB[rv.slot], rv.phase, 4000000);
          rv.next();
        }
      }
    } else if (warp < DW + 2 * SETS) {
      // ------------------------------ MMAs ------------------------------
      const int set = warp - DW - SETS;
      const uint32_t smA = smA0 + set * (g.nA * SEG * SA), smB = smB0 + (STAGE == 2 ? set * (g.nB * SEG * SB) : 0);
      const uint32_t ts = tm + set * SETC;
      Ring ra(g.nA), rb(STAGE == 2 ? g.nB : g.tasksB);
      int n = 0, fills = 0;  // fills of the sets, of this set
      bool ok = true;
      for (int ti = blockIdx.x; ti < g.ntasks && ok; ti += gridDim.x) {
        Job<NS, STAGE> job;
        job.init(g, g.tasks[ti]);
        const int noct = __shfl_sync(0xffffffffu, job.noct, 0);
        const uint32_t id = idesc_f16(16 * noct);
        const uint32_t bstep = 512u * noct;  // one plane of one K step
        if (STAGE != 2 && !bwait(&fullB[rb.slot], rb.phase)) { ok = false; break; }
        const uint32_t bt = smB + rb.slot * (g.nB * SB);
        for (int m0 = 0; m0 < job.outer && ok; m0 += job.G) {
          const int Gm = min(job.G, job.outer - m0);
          int r = (n ^ set) & (SETS - 1);
          n += job.R;
          OzRnd nx = job.round(r);
          for (; r < job.R && ok; r += SETS, ++fills) {
            const int nks = __shfl_sync(0xffffffffu, nx.nks, 0);
            nx = job.round(r + SETS);
            const Ring rr = rb;
            if constexpr (NS == 6) {  // per row tile the high classes, then the low ones; its K steps stay in the ring
              if (fills >= 1 && !bwait(&tfreeH, (fills - 1) & 1)) { ok = false; break; }
              for (int gi = 0; gi < Gm && ok; ++gi) {
                if (STAGE == 2) rb = rr;
                const uint32_t d0 = ts + (uint32_t)(gi * 16 * noct);
                const Ring a1 = ra, b1 = rb;
                auto bat = [&](int ks) { return STAGE == 2 ? smB + rb.slot * SB : bt + (r * OCT + ks) * NS * bstep; };
                for (int ks = 0; ks < nks; ++ks) {
                  if (!bwait(&full[set][ra.slot], ra.phase)) { ok = false; break; }
                  tc::fence_after_sync();
                  if (elect_one()) oz_mmas<NS, 4, OzCfg<NS>::CMAX>(d0, smA + ra.slot * SA, bat(ks), bstep, id, ks > 0);
                  __syncwarp();
                  ra.next();
                  if (STAGE == 2) rb.next();
                }
                if (!ok) break;
                if (gi == Gm - 1 && elect_one()) tc::commit(&doneH);
                __syncwarp();
                if (gi == 0 && fills >= 1 && !bwait(&tfree[set], (fills - 1) & 1)) { ok = false; break; }
                ra = a1;
                rb = b1;
                for (int ks = 0; ks < nks; ++ks) {
                  if (elect_one()) {
                    oz_mmas<NS, 0, 3>(d0, smA + ra.slot * SA, bat(ks), bstep, id, ks > 0);
                    tc::commit(&emptyA[set][ra.slot]);
                    if (STAGE == 2 && gi == Gm - 1) tc::commit(&emptyB[set][rb.slot]);
                  }
                  __syncwarp();
                  ra.next();
                  if (STAGE == 2) rb.next();
                }
              }
            } else {
              if (fills >= 1 && !bwait(&tfree[set], (fills - 1) & 1)) { ok = false; break; }
              for (int gi = 0; gi < Gm && ok; ++gi) {
                if (STAGE == 2) rb = rr;
                const uint32_t d0 = ts + (uint32_t)(gi * 16 * noct);
                for (int ks = 0; ks < nks; ks += SEG) {
                  if (!bwait(&full[set][ra.slot], ra.phase)) { ok = false; break; }
                  tc::fence_after_sync();
                  const uint32_t a0 = smA + ra.slot * (SEG * SA);
                  const uint32_t b0 = STAGE == 2 ? smB + rb.slot * (SEG * SB) : bt + (r * OCT + ks) * NS * bstep;
                  if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < SEG; ++k) {
                      if (ks + k >= nks) break;
                      oz_mmas<NS, 0, OzCfg<NS>::CMAX>(d0, a0 + k * SA, b0 + k * NS * bstep, bstep, id, ks + k > 0 ? 1u : 0u);
                    }
                    tc::commit(&emptyA[set][ra.slot]);
                    if (STAGE == 2 && gi == Gm - 1) tc::commit(&emptyB[set][rb.slot]);
                  }
                  __syncwarp();
                  ra.next();
                  if (STAGE == 2) rb.next();
                }
              }
            }
            if (!ok) break;
            if (elect_one()) tc::commit(&done[set]);
            __syncwarp();
          }
        }
        if (STAGE != 2) {
          if (!ok) break;
          if (elect_one()) tc::commit(&emptyB[0][rb.slot]);
          __syncwarp();
          rb.next();
        }
      }
      if (elect_one()) tc::commit(&last);  // arrives when every MMA issued above has completed
      __syncwarp();
    }
  }
  __syncthreads();
  if (tid == 0) tc::mbar_wait(&last, 0u, 4000000);  // every issued MMA has completed
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tm, 512);
}

// The six digits of x relative to 2^E, |x| < 2^E, from its bits: x 2^(60-E) as a 64-bit integer
// (rounded towards zero: below 2^(E-60)), digits of 9 bits from the top, the last one with 7 bits of
// fraction.  Infinities and NaN give NaN.
__device__ __forceinline__ void double_digits(double x, int e2, float (&s)[6]) {
  const long long b = __double_as_longlong(x);
  const int be = (int)((b >> 52) & 0x7ff);
  long long m = b & 0xfffffffffffffll;
  if (be) m |= 1ll << 52;
  const int sh = e2 + 1022 - max(be, 1);  // x = m 2^(max(be, 1) - 1075): F = m 2^(7 - sh)
  long long F = sh <= 7 ? m << (7 - sh) : sh < 64 ? m >> (sh - 7) : 0ll;
  if (b < 0) F = -F;
  auto digit = [](int d) { return __int_as_float(0x4b400000 + d) - 12582912.f; };  // |d| < 2^22, exact
#pragma unroll
  for (int p = 0; p < 5; ++p) {
    const int k = 52 - 9 * p;
    const int d = (int)((F + (1ll << (k - 1))) >> k);
    F -= (long long)d << k;
    s[p] = digit(d);
  }
  s[5] = digit((int)F) * 0x1p-7f;
  if (be == 0x7ff) s[0] = __int_as_float(0x7fffffff);
}

// Element k of row source s of an image (zero outside).
__device__ __forceinline__ double2 load(const double2 *__restrict__ s, const OzBuild &t, bool rv, int k,
                                        const double *__restrict__ scale) {
  double2 v = make_double2(0.0, 0.0);
  const int k1 = k / t.kd, k0 = k - k1 * t.kd;
  if (rv && k0 < t.kv && k1 < t.kn) {
    v = s[k1 * t.ks1 + (int64_t)k0 * t.ks0];
    if (t.conj) v.y = -v.y;
    if (t.kx >= 0) {
      const double f = scale[t.kx + k];
      v = make_double2(v.x * f, v.y * f);
    }
  }
  return v;
}

// Operand images from FP64 data: one CTA per image, OCT lanes per row (one
// octet each), the row's exponent by a shuffle over them.
template <int NS>
__global__ void __launch_bounds__(128) oz_build_kernel(const OzBuild *__restrict__ tasks,
                                                       const double2 *__restrict__ src, char *__restrict__ dst,
                                                       const double *__restrict__ scale_k) {
  constexpr int OCT = OzCfg<NS>::OCT;
  const OzBuild t = tasks[blockIdx.x];
  const int q = threadIdx.x % OCT;
  const int nks = t.nks;
  char *blob = dst + t.dst;
  const int64_t pstride = t.isb ? 64 * t.rows : 4096;  // one K step of one plane
  for (int lr = threadIdx.x / OCT; lr < t.rows; lr += 128 / OCT) {
    const int r = t.r0 + lr, r1 = r / t.rd, r0 = r - r1 * t.rd;
    const bool rv = r0 < t.rv && r1 < t.rn && q < nks;
    const double2 *s = src + t.src + r1 * t.rs1 + (int64_t)r0 * t.rs0;
    double2 v[8];
    int e2;        // the row's exponent
    float f = 0.f, m1 = 0.f, scale;
    if constexpr (NS == 3) {
      float m = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        v[e] = load(s, t, rv, 8 * q + e, scale_k);
        m = fmaxf(m, fmaxf(fabsf((float)v[e].x), fabsf((float)v[e].y)));
      }
#pragma unroll
      for (int d = 1; d < OCT; d <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
      e2 = oz_exponent(m);
      f = oz_pow2(15 - e2);
      m1 = oz_m1(nks);
      scale = oz_pow2(e2 - 15);
    } else {
      // FP64's own exponent range, by integer operations (the FP64 pipe is 64 times slower)
      int be = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        v[e] = load(s, t, rv, 8 * q + e, scale_k);
        const int hx = __double2hiint(v[e].x) & 0x7fffffff, hy = __double2hiint(v[e].y) & 0x7fffffff;
        // subnormal numbers have the smallest normal number's exponent; zero has none
        be = max(be, max(hx >> 20, hy >> 20));
        if ((hx | hy | __double2loint(v[e].x) | __double2loint(v[e].y)) != 0) be = max(be, 1);
      }
#pragma unroll
      for (int d = 1; d < OCT; d <<= 1) be = max(be, __shfl_xor_sync(0xffffffffu, be, d));
      e2 = be - 1022;
      scale = __int_as_float((be ? e2 : -OZ_ELIM) - 8);
    }
    if (q < nks) {
      uint32_t w[NS][8];
      F2 sl[8][NS];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if constexpr (NS == 3) {
          const F2 h{(float)v[e].x, (float)v[e].y};
          const F2 l{(float)(v[e].x - (double)h.x), (float)(v[e].y - (double)h.y)};
          oz_slice(h, l, h, both(f), both(m1), sl[e]);
        } else {
          float sr[6], si[6];
          double_digits(v[e].x, e2, sr);
          double_digits(v[e].y, e2, si);
#pragma unroll
          for (int p = 0; p < NS; ++p) sl[e][p] = {sr[p], si[p]};
        }
      }
      if (!t.isb) {
#pragma unroll
        for (int p = 0; p < NS; ++p) {
#pragma unroll
          for (int e = 0; e < 8; ++e) w[p][e] = h2(sl[e][p]);
          st_octet(blob + (q * NS + p) * pstride + lr * 32, w[p], (lr >> 2) & 1);
        }
      } else {  // rows (n, 0) = [Br -Bi], (n, 1) = [Bi Br]
#pragma unroll
        for (int p = 0; p < NS; ++p) {
          char *o = blob + (q * NS + p) * pstride + lr * 64;
#pragma unroll
          for (int e = 0; e < 8; ++e) w[p][e] = h2({sl[e][p].x, -sl[e][p].y});
          st_octet(o, w[p], (lr >> 1) & 1);
#pragma unroll
          for (int e = 0; e < 8; ++e) w[p][e] = h2({sl[e][p].y, sl[e][p].x});
          st_octet(o + 32, w[p], (lr >> 1) & 1);
        }
      }
      if (q == 0) reinterpret_cast<float *>(blob + NS * nks * pstride)[lr] = scale;
    }
  }
}

// One CTA per row (launch_oz_row_scale).  Bound: reading X once, 10 us where the transform takes 100.
__global__ void __launch_bounds__(1024) oz_row_scale_kernel(const TSlab *__restrict__ slabs, int nslabs,
                                                            const double2 *__restrict__ X, int row0, int nin,
                                                            double *__restrict__ scale) {
  __shared__ int part[32];
  const int i = blockIdx.x;
  int m = 0;  // upper word of the largest finite component, at least 1 if there is one but zero
  auto word = [](double v) {
    const int h = __double2hiint(v) & 0x7fffffff;
    return h >= 0x7ff00000 ? 0 : h ? h : __double2loint(v) ? 1 : 0;
  };
  // chunks of 128 columns dealt to the warps over all slabs: small slabs are read side by side (54 of 89 columns: 8 us less
  // of a Dyson pass's 0.245 ms of transforms than one after the other)
  const int lane = threadIdx.x & 31;
  int first = threadIdx.x >> 5;  // this warp's first chunk of the slab, modulo 32
  for (int s = 0; s < nslabs; ++s) {
    const TSlab sl = slabs[s];
    const double2 *x = X + sl.x + (int64_t)(row0 + i) * sl.ldx;
    const int chunks = (sl.ncols + 127) >> 7;
    for (int k = first & 31; k < chunks; k += 32) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = k * 128 + j * 32 + lane;
        const double2 v = c < sl.ncols ? x[c] : make_double2(0.0, 0.0);
        m = max(m, max(word(v.x), word(v.y)));
      }
    }
    first -= chunks;
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = __reduce_max_sync(0xffffffffu, part[threadIdx.x]);
    if (threadIdx.x == 0) {
      const int e = min(max((m >> 20) - 1022, -500), 500);
      scale[i] = m ? __hiloint2double((1023 - e) << 20, 0) : 1.0;
      scale[nin + i] = m ? __hiloint2double((1023 + e) << 20, 0) : 0.0;
    }
  }
}

}  // namespace

template <int NS>
static void set_attributes() {
  for (auto k : {oz_gemm_kernel<NS, 0, false>, oz_gemm_kernel<NS, 0, true>, oz_gemm_kernel<NS, 1, false>,
                 oz_gemm_kernel<NS, 1, true>, oz_gemm_kernel<NS, 2, false>})
    GWGB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
}

void set_oz_kernel_attributes() {
  set_attributes<3>();
  set_attributes<6>();
}

// Stages 1 and 2 hold the column operand of a task (max_kos K steps) and, where that leaves room
// for three segments of A, that of the next; stage 3 streams both operands.
void oz_rings(int ns, int stage, int max_kos, OzArgs *a) {
  const int seg = ns == 3 ? (stage == 2 ? OzCfg<3>::SEG3 : OzCfg<3>::SEG)
                          : (stage == 2 ? OzCfg<6>::SEG3 : OzCfg<6>::SEG);
  const int slotA = seg * ns * 4096, stepB = ns * 512 * OZ_OCT;
  const int sets = ns == 3 ? OzCfg<3>::SETS : OzCfg<6>::SETS;
  if (stage == 2) {
    a->nA = a->nB = std::min(OZ_RING, OZ_SMEM / (sets * (slotA + seg * stepB)));
  } else {
    a->nB = max_kos;
    auto ring = [&](int tasks) { return std::min(OZ_RING, (OZ_SMEM - tasks * a->nB * stepB) / (sets * slotA)); };
    a->tasksB = ring(2) >= (ns == 6 ? OZ_OCT : 3) ? 2 : 1;  // six slices hold a round of A
    a->nA = ring(a->tasksB);
  }
  GWGB_REQUIRE(a->nA >= (ns == 6 ? OZ_OCT : 2), GWGB_E_UNSUPPORTED, "sliced GEMM rings too small");
}

template <int NS>
static void launch(int stage, bool multi, const OzArgs &a, int grid, cudaStream_t st) {
  auto k = stage == 0 ? (multi ? oz_gemm_kernel<NS, 0, true> : oz_gemm_kernel<NS, 0, false>)
           : stage == 1 ? (multi ? oz_gemm_kernel<NS, 1, true> : oz_gemm_kernel<NS, 1, false>)
                        : oz_gemm_kernel<NS, 2, false>;
  k<<<grid, oz_threads<NS>, OZ_SMEM, st>>>(a);
}

void launch_oz_gemm(int ns, int stage, bool multi, const OzArgs &a, int nsm, cudaStream_t st) {
  if (a.ntasks == 0) return;
  const int grid = std::min(a.ntasks, std::max(1, nsm));
  if (ns == 3)
    launch<3>(stage, multi, a, grid, st);
  else
    launch<6>(stage, multi, a, grid, st);
  GWGB_CUDA(cudaGetLastError());
}

void launch_oz_row_scale(const TSlab *slabs, int nslabs, const double2 *X, int row0, int nin, double *scale,
                         cudaStream_t st) {
  oz_row_scale_kernel<<<nin, 1024, 0, st>>>(slabs, nslabs, X, row0, nin, scale);
  GWGB_CUDA(cudaGetLastError());
}

void launch_oz_build(int ns, const OzBuild *tasks, int64_t ntasks, const double2 *src, char *dst, cudaStream_t st,
                     const double *scale) {
  if (ntasks == 0) return;
  if (ns == 3)
    oz_build_kernel<3><<<(unsigned)ntasks, 128, 0, st>>>(tasks, src, dst, scale);
  else
    oz_build_kernel<6><<<(unsigned)ntasks, 128, 0, st>>>(tasks, src, dst, scale);
  GWGB_CUDA(cudaGetLastError());
}

}  // namespace gwgb

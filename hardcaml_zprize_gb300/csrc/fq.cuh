// Base field of BLS12-377 (q, 377 bits) on sm_103a: twelve 32-bit limbs, Montgomery form with
// R = 2^384 -- the same R as arkworks' six 64-bit limbs, so a device element is bit-for-bit the
// arkworks Fq representation once it is fully reduced.
//
// Values are kept "lazy" in [0, 2q): 4q < 2^384, so the CIOS product of two such values is again
// below 2q without a final subtraction.  Addition/subtraction reduce by 2q.  fq_canon() brings a
// value to [0, q) for comparisons and for the ABI.
//
// The multiplier is operand-scanning CIOS with 32 x 32 + 64 -> 64 wide multiplies in carry chains:
// 12 + 11 limb products per row (q's lowest limb is 1), 276 wide IMADs per product.  The algorithmic count for
// the roofline stays 588 32-bit IMAD per product (lo and hi halves of 12 x 12 + 12 x 12).
// The field is the one the reference computes in with GMP (host/msm_compute/include/
// bls12_377_g1/bls12_377_g1.h:31-33, 90-219); the limb layout is new.
#pragma once
#include <stdint.h>

#include "fq_divstep.cuh"

#define FQ_LIMBS 12

// q, 2q and 4q, little-endian 32-bit limbs
#define BLS_Q {0x00000001u, 0x8508c000u, 0x30000000u, 0x170b5d44u, 0xba094800u, 0x1ef3622fu, 0x00f5138fu, 0x1a22d9f3u, 0x6ca1493bu, 0xc63b05c0u, 0x17c510eau, 0x01ae3a46u}
#define BLS_Q2 {0x00000002u, 0x0a118000u, 0x60000001u, 0x2e16ba88u, 0x74129000u, 0x3de6c45fu, 0x01ea271eu, 0x3445b3e6u, 0xd9429276u, 0x8c760b80u, 0x2f8a21d5u, 0x035c748cu}
#define BLS_Q4 {0x00000004u, 0x14230000u, 0xc0000002u, 0x5c2d7510u, 0xe8252000u, 0x7bcd88beu, 0x03d44e3cu, 0x688b67ccu, 0xb28524ecu, 0x18ec1701u, 0x5f1443abu, 0x06b8e918u}
// -q^-1 mod 2^32 (q = 1 mod 2^46)
#define BLS_QINV 0xffffffffu
// Montgomery-form constants (value * 2^384 mod q)
#define BLS_ONE {0xffffff68u, 0x02cdffffu, 0x7fffffb1u, 0x51409f83u, 0x8a7d3ff2u, 0x9f7db3a9u, 0x6e7c6305u, 0x7b4e97b7u, 0x803c84e8u, 0x4cf495bfu, 0xe2fdf49au, 0x008d6661u}
#define BLS_INV2 {0xffffffb4u, 0x8166ffffu, 0xbfffffd8u, 0x28a04fc1u, 0xc53e9ff9u, 0xcfbed9d4u, 0xb73e3182u, 0x3da74bdbu, 0xc01e4274u, 0x267a4adfu, 0xf17efa4du, 0x0046b330u}
// twisted Edwards k = 2d and d (bls12_377_g1.h:37-39, 46-48)
#define BLS_TE_K {0xbb58e892u, 0x33f6817bu, 0xff054e5du, 0x3fd664cau, 0xd6752edau, 0x6ad7181au, 0x47ff7cfeu, 0x55eabefau, 0x93fe9656u, 0xacf17111u, 0x199ed6ffu, 0x008d1a81u}
#define BLS_TE_D {0xddac7449u, 0x99fb40bdu, 0x7f82a72eu, 0x1feb3265u, 0x6b3a976du, 0x356b8c0du, 0x23ffbe7fu, 0x2af55f7du, 0xc9ff4b2bu, 0xd678b888u, 0x8ccf6b7fu, 0x00468d40u}
// Weierstrass -> Montgomery scale s (bls12_377_g1.h:40-42) and the twisted scale (:34-36)
#define BLS_WS {0x27ce5f5fu, 0x171ef565u, 0x214ae372u, 0x6e5b6922u, 0x26a8cea6u, 0xc47c7b6au, 0x2d74b055u, 0xc22f509cu, 0xcbda4b0au, 0x0134cecbu, 0x229913d6u, 0x001ef3f3u}
#define BLS_TWISTED_SCALE {0xe4aeaf1eu, 0x432a25c1u, 0xcd4c9661u, 0x5b39d21fu, 0xcd09455du, 0x692669ecu, 0x0f74f6bbu, 0xddae3345u, 0xabb65d37u, 0x76cbfeebu, 0x517df4cdu, 0x0143462fu}
// 1/c_B and c_A/(3 c_B) of the Montgomery -> Weierstrass map (bls12_377_g1.h:366-374)
#define BLS_INV_CB {0x776b1e1du, 0x455ce02fu, 0x63e0aa56u, 0x4b123b66u, 0x73fa6bf3u, 0x4d75723eu, 0x885e1101u, 0x468df1d4u, 0x638ee120u, 0x039e6c63u, 0x67cb3b82u, 0x005cdbd9u}
#define BLS_CA_OVER_3CB {0x00000099u, 0x823ac000u, 0xb000004fu, 0xc5cabdc0u, 0x2f8c080du, 0x7f75ae86u, 0x9278b089u, 0x9ed4423bu, 0xec64c452u, 0x79467000u, 0x34c71c50u, 0x0120d3e4u}
// (1/c_B) R^3 and ts (1/c_B) R^3, factors of numerators that meet a plain inverse (te_to_weierstrass_warp)
#define BLS_INV_CB_R3X {0xa53f9bdfu, 0xe50fb361u, 0x8a41d16bu, 0x7c0b9d21u, 0xf62d549bu, 0x87b97febu, 0xa7d11b60u, 0x8ddcefe4u, 0x334f01a9u, 0xe403bc7au, 0x816dd8dbu, 0x002693d5u}
#define BLS_TS_INV_CB_R3X {0x8249903fu, 0x89d5d01eu, 0xd7a74139u, 0x80a3ad71u, 0xa655ae9fu, 0xd0ecc29bu, 0xb333f4c5u, 0x45a17a34u, 0x4d6653fbu, 0x556d2dacu, 0x17c7aa65u, 0x000e207au}
// R^3 mod q: turns a plain inverse of a Montgomery-form value into the Montgomery-form inverse
#define BLS_R3 {0x8815de20u, 0x581f532fu, 0xbe329585u, 0xe50f4148u, 0x0449f513u, 0x2be8b118u, 0xc804a20eu, 0x6a2a9516u, 0x13590cb9u, 0x3f725407u, 0xc0e7dda5u, 0x01065ab4u}
// q - 2, the Fermat inversion exponent
#define BLS_QM2 {0xffffffffu, 0x8508bfffu, 0x30000000u, 0x170b5d44u, 0xba094800u, 0x1ef3622fu, 0x00f5138fu, 0x1a22d9f3u, 0x6ca1493bu, 0xc63b05c0u, 0x17c510eau, 0x01ae3a46u}

struct fq_t {
  uint32_t v[FQ_LIMBS];
};

// ---- carry-chain primitives (one PTX instruction each; the carry flag lives between them) ----
__device__ __forceinline__ uint32_t add_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t addc_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t addc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("addc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t sub_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t subc_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t subc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("subc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// ---- constructors ----
__device__ __forceinline__ fq_t fq_from(const uint32_t (&c)[FQ_LIMBS]) {
  fq_t r;
#pragma unroll
  for (int i = 0; i < FQ_LIMBS; i++) r.v[i] = c[i];
  return r;
}
__device__ __forceinline__ fq_t fq_zero() {
  fq_t r;
#pragma unroll
  for (int i = 0; i < FQ_LIMBS; i++) r.v[i] = 0;
  return r;
}
__device__ __forceinline__ fq_t fq_one() {
  const uint32_t c[FQ_LIMBS] = BLS_ONE;
  return fq_from(c);
}

// ---- a * b * 2^-384 mod q (CIOS; inputs and output in [0, 2q)) ----
// The steps are CIOS (Koc, Acar, Kaliski, "Analyzing and Comparing Montgomery Multiplication Algorithms", IEEE
// Micro 1996) with the even and the odd columns kept as two carry chains, the published arrangement for 32-bit
// GPU multipliers (Emmart, Luitjens, Weems, Woolley, "Optimizing Modular Multiplication for NVIDIA's Maxwell
// GPUs", ARITH 2016).
// Row i adds b_i a and then m q to the running value and drops its lowest word, m = -t0 (q = 1 mod
// 2^32 and -q^-1 = -1 mod 2^32, so the row factor needs no product and m q0 + t0 = 0 with a carry of
// (t0 != 0)).  The running value is the sum of two word vectors on 64-bit lanes: E, words 0 to 11,
// takes the products of the even words of a (and q), O, words 1 to 12, those of the odd ones.  All
// lanes of a vector are one carry chain of mad.lo.cc / madc.hi.cc pairs, and ptxas makes each pair
// one wide multiply with a 64-bit addend, carry in and carry out.  Dropping word 0 swaps the two
// vectors' roles: O becomes the new E, the old E moves down two words and becomes the new O, and its
// word 1 is added to the new E's word 0 on the way (that carry starts the new O's chain).
//
// The negation of t0 is written as ~t0 + 1: ptxas folds a plain negation into the products of m and
// then splits each pair of that chain into a low and a high multiply (ncu opcode counts: 144 wide
// multiplies and 132 pairs; with it written so, 276 wide multiplies, 42 + 31 carry adds, 12 LOP3,
// 36 moves).  What bounds it is the multiply pipe: a wide multiply holds it four cycles, 1104 of
// about 1195 cycles per warp-product.  Products/s on GB300 in a chain of products (mixed adds/s in
// k_accumulate's loop): wide multiplies without addend and four carry chains per row, the form
// before, 2.18e10 (3.01e9); this one with the pairs of m split 2.61e10 (3.61e9); this one 3.12e10
// (4.25e9); 13 signed 30-bit limbs with 64-bit accumulators and no carry chains 2.46e10 (3.44e9).
// Bound: at the start of a row t < 4q < 2^384, and no row sum leaves 13 words, for any a < 2^383
// and any b; so O, which is at most the sum, has no carry out of its top word.
struct fq_lanes {  // six 64-bit lanes
  uint32_t w[FQ_LIMBS];
};

// x += sum over k of a[k] b at lane k, carry out added to top.  In these four every output is written before
// the last input is read: all are early clobbers.
__device__ __forceinline__ void fq_chain(fq_lanes &x, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t a4, uint32_t a5, uint32_t b, uint32_t &top) {
  asm("mad.lo.cc.u32 %0, %13, %19, %0;\n\tmadc.hi.cc.u32 %1, %13, %19, %1;\n\t"
      "madc.lo.cc.u32 %2, %14, %19, %2;\n\tmadc.hi.cc.u32 %3, %14, %19, %3;\n\t"
      "madc.lo.cc.u32 %4, %15, %19, %4;\n\tmadc.hi.cc.u32 %5, %15, %19, %5;\n\t"
      "madc.lo.cc.u32 %6, %16, %19, %6;\n\tmadc.hi.cc.u32 %7, %16, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %17, %19, %8;\n\tmadc.hi.cc.u32 %9, %17, %19, %9;\n\t"
      "madc.lo.cc.u32 %10, %18, %19, %10;\n\tmadc.hi.cc.u32 %11, %18, %19, %11;\n\t"
      "addc.u32 %12, %12, 0;"
      : "+&r"(x.w[0]), "+&r"(x.w[1]), "+&r"(x.w[2]), "+&r"(x.w[3]), "+&r"(x.w[4]), "+&r"(x.w[5]), "+&r"(x.w[6]),
        "+&r"(x.w[7]), "+&r"(x.w[8]), "+&r"(x.w[9]), "+&r"(x.w[10]), "+&r"(x.w[11]), "+&r"(top)
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(a4), "r"(a5), "r"(b));
}
// the same without a carry out
__device__ __forceinline__ void fq_chain_end(fq_lanes &x, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t a4, uint32_t a5, uint32_t b) {
  asm("mad.lo.cc.u32 %0, %12, %18, %0;\n\tmadc.hi.cc.u32 %1, %12, %18, %1;\n\t"
      "madc.lo.cc.u32 %2, %13, %18, %2;\n\tmadc.hi.cc.u32 %3, %13, %18, %3;\n\t"
      "madc.lo.cc.u32 %4, %14, %18, %4;\n\tmadc.hi.cc.u32 %5, %14, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %15, %18, %6;\n\tmadc.hi.cc.u32 %7, %15, %18, %7;\n\t"
      "madc.lo.cc.u32 %8, %16, %18, %8;\n\tmadc.hi.cc.u32 %9, %16, %18, %9;\n\t"
      "madc.lo.cc.u32 %10, %17, %18, %10;\n\tmadc.hi.u32 %11, %17, %18, %11;"
      : "+&r"(x.w[0]), "+&r"(x.w[1]), "+&r"(x.w[2]), "+&r"(x.w[3]), "+&r"(x.w[4]), "+&r"(x.w[5]), "+&r"(x.w[6]),
        "+&r"(x.w[7]), "+&r"(x.w[8]), "+&r"(x.w[9]), "+&r"(x.w[10]), "+&r"(x.w[11])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(a4), "r"(a5), "r"(b));
}
// e0 += s, then lanes 0 to 4 of x and a new lane 5 (from zero) take the products, the sum's carry first
__device__ __forceinline__ void fq_chain_shifted(fq_lanes &x, uint32_t &e0, uint32_t s, uint32_t a0, uint32_t a1,
                                                 uint32_t a2, uint32_t a3, uint32_t a4, uint32_t a5, uint32_t b) {
  asm("add.cc.u32 %12, %12, %20;\n\t"
      "madc.lo.cc.u32 %0, %13, %19, %0;\n\tmadc.hi.cc.u32 %1, %13, %19, %1;\n\t"
      "madc.lo.cc.u32 %2, %14, %19, %2;\n\tmadc.hi.cc.u32 %3, %14, %19, %3;\n\t"
      "madc.lo.cc.u32 %4, %15, %19, %4;\n\tmadc.hi.cc.u32 %5, %15, %19, %5;\n\t"
      "madc.lo.cc.u32 %6, %16, %19, %6;\n\tmadc.hi.cc.u32 %7, %16, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %17, %19, %8;\n\tmadc.hi.cc.u32 %9, %17, %19, %9;\n\t"
      "madc.lo.cc.u32 %10, %18, %19, 0;\n\tmadc.hi.u32 %11, %18, %19, 0;"
      : "+&r"(x.w[0]), "+&r"(x.w[1]), "+&r"(x.w[2]), "+&r"(x.w[3]), "+&r"(x.w[4]), "+&r"(x.w[5]), "+&r"(x.w[6]),
        "+&r"(x.w[7]), "+&r"(x.w[8]), "+&r"(x.w[9]), "=&r"(x.w[10]), "=&r"(x.w[11]), "+&r"(e0)
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(a4), "r"(a5), "r"(b), "r"(s));
}
// x += m (1 + sum over k >= 1 of a[k] 2^64k), word 0 becomes zero (m = -x.w[0]), carry out added to top
__device__ __forceinline__ void fq_chain_reduce(fq_lanes &x, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t a4,
                                                uint32_t a5, uint32_t m, uint32_t &top) {
  asm("{\n\t.reg .u32 z;\n\tadd.cc.u32 z, %0, %18;\n\taddc.cc.u32 %1, %1, 0;\n\t"
      "madc.lo.cc.u32 %2, %13, %18, %2;\n\tmadc.hi.cc.u32 %3, %13, %18, %3;\n\t"
      "madc.lo.cc.u32 %4, %14, %18, %4;\n\tmadc.hi.cc.u32 %5, %14, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %15, %18, %6;\n\tmadc.hi.cc.u32 %7, %15, %18, %7;\n\t"
      "madc.lo.cc.u32 %8, %16, %18, %8;\n\tmadc.hi.cc.u32 %9, %16, %18, %9;\n\t"
      "madc.lo.cc.u32 %10, %17, %18, %10;\n\tmadc.hi.cc.u32 %11, %17, %18, %11;\n\t"
      "addc.u32 %12, %12, 0;\n\t}"
      : "+&r"(x.w[0]), "+&r"(x.w[1]), "+&r"(x.w[2]), "+&r"(x.w[3]), "+&r"(x.w[4]), "+&r"(x.w[5]), "+&r"(x.w[6]),
        "+&r"(x.w[7]), "+&r"(x.w[8]), "+&r"(x.w[9]), "+&r"(x.w[10]), "+&r"(x.w[11]), "+&r"(top)
      : "r"(a1), "r"(a2), "r"(a3), "r"(a4), "r"(a5), "r"(m));
}
// -x, kept apart from the products that use it (see above)
__device__ __forceinline__ uint32_t fq_row_factor(uint32_t x) {
  uint32_t m;
  asm("{\n\t.reg .u32 t;\n\tnot.b32 t, %1;\n\tadd.u32 %0, t, 1;\n\t}" : "=r"(m) : "r"(x));
  return m;
}

__device__ __forceinline__ fq_t fq_mul(const fq_t &x, const fq_t &y) {
  const uint32_t q[FQ_LIMBS] = BLS_Q;
  const uint32_t *a = x.v;
  fq_lanes E, O;
#pragma unroll
  for (int i = 0; i < FQ_LIMBS; i++) {
    const uint32_t b = y.v[i];
    if (i == 0) {
#pragma unroll
      for (int j = 0; j < FQ_LIMBS; j += 2) {
        const uint64_t e = (uint64_t)a[j] * b, o = (uint64_t)a[j + 1] * b;
        E.w[j] = (uint32_t)e;
        E.w[j + 1] = (uint32_t)(e >> 32);
        O.w[j] = (uint32_t)o;
        O.w[j + 1] = (uint32_t)(o >> 32);
      }
    } else {
      fq_lanes N;  // the old E, two words down
#pragma unroll
      for (int k = 0; k < FQ_LIMBS - 2; k++) N.w[k] = E.w[k + 2];
      const uint32_t s = E.w[1];
      E = O;
      fq_chain_shifted(N, E.w[0], s, a[1], a[3], a[5], a[7], a[9], a[11], b);
      O = N;
      fq_chain(E, a[0], a[2], a[4], a[6], a[8], a[10], b, O.w[11]);
    }
    const uint32_t m = fq_row_factor(E.w[0]);
    fq_chain_end(O, q[1], q[3], q[5], q[7], q[9], q[11], m);
    fq_chain_reduce(E, q[2], q[4], q[6], q[8], q[10], m, O.w[11]);
  }
  fq_t r;  // E without its zero word 0, plus O
  r.v[0] = add_cc(O.w[0], E.w[1]);
#pragma unroll
  for (int k = 1; k < FQ_LIMBS - 1; k++) r.v[k] = addc_cc(O.w[k], E.w[k + 1]);
  r.v[FQ_LIMBS - 1] = addc(O.w[FQ_LIMBS - 1], 0u);
  return r;
}

__device__ __forceinline__ fq_t fq_sqr(const fq_t &a) { return fq_mul(a, a); }

// r = x - 2q if x >= 2q else x   (x < 4q < 2^384)
__device__ __forceinline__ fq_t fq_reduce_2q(const uint32_t (&x)[FQ_LIMBS]) {
  const uint32_t q2[FQ_LIMBS] = BLS_Q2;
  uint32_t d[FQ_LIMBS];
  d[0] = sub_cc(x[0], q2[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS; j++) d[j] = subc_cc(x[j], q2[j]);
  const uint32_t borrow = subc(0u, 0u);  // 0xffffffff if x < 2q
  fq_t r;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) r.v[j] = borrow ? x[j] : d[j];
  return r;
}

__device__ __forceinline__ fq_t fq_add(const fq_t &a, const fq_t &b) {
  uint32_t s[FQ_LIMBS];
  s[0] = add_cc(a.v[0], b.v[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS - 1; j++) s[j] = addc_cc(a.v[j], b.v[j]);
  s[FQ_LIMBS - 1] = addc(a.v[FQ_LIMBS - 1], b.v[FQ_LIMBS - 1]);
  return fq_reduce_2q(s);
}

__device__ __forceinline__ fq_t fq_sub(const fq_t &a, const fq_t &b) {
  const uint32_t q2[FQ_LIMBS] = BLS_Q2;
  uint32_t d[FQ_LIMBS];
  d[0] = sub_cc(a.v[0], b.v[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS; j++) d[j] = subc_cc(a.v[j], b.v[j]);
  const uint32_t mask = subc(0u, 0u);  // all ones on borrow
  fq_t r;
  r.v[0] = add_cc(d[0], q2[0] & mask);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS - 1; j++) r.v[j] = addc_cc(d[j], q2[j] & mask);
  r.v[FQ_LIMBS - 1] = addc(d[FQ_LIMBS - 1], q2[FQ_LIMBS - 1] & mask);
  return r;
}

// Unreduced forms for operands that only feed products: for a, b < 2q, a + b and a - b + 2q are
// below 4q, and a product of two values below 8q is below q + 64 q (q / 2^384) < 1.5q.
__device__ __forceinline__ fq_t fq_add_lazy(const fq_t &a, const fq_t &b) {
  fq_t r;
  r.v[0] = add_cc(a.v[0], b.v[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS - 1; j++) r.v[j] = addc_cc(a.v[j], b.v[j]);
  r.v[FQ_LIMBS - 1] = addc(a.v[FQ_LIMBS - 1], b.v[FQ_LIMBS - 1]);
  return r;
}
__device__ __forceinline__ fq_t fq_sub_lazy(const fq_t &a, const fq_t &b) {
  const uint32_t q2[FQ_LIMBS] = BLS_Q2;
  uint32_t d[FQ_LIMBS];
  d[0] = add_cc(a.v[0], q2[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS; j++) d[j] = addc_cc(a.v[j], q2[j]);
  fq_t r;
  r.v[0] = sub_cc(d[0], b.v[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS - 1; j++) r.v[j] = subc_cc(d[j], b.v[j]);
  r.v[FQ_LIMBS - 1] = subc(d[FQ_LIMBS - 1], b.v[FQ_LIMBS - 1]);
  return r;
}

// a - b + 4q, b below 4q
__device__ __forceinline__ fq_t fq_sub_lazy4(const fq_t &a, const fq_t &b) {
  const uint32_t q4[FQ_LIMBS] = BLS_Q4;
  fq_t r;
  r.v[0] = add_cc(a.v[0], q4[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS; j++) r.v[j] = addc_cc(a.v[j], q4[j]);
  r.v[0] = sub_cc(r.v[0], b.v[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS - 1; j++) r.v[j] = subc_cc(r.v[j], b.v[j]);
  r.v[FQ_LIMBS - 1] = subc(r.v[FQ_LIMBS - 1], b.v[FQ_LIMBS - 1]);
  return r;
}
// a 2^s, s = 0 or 1
__device__ __forceinline__ fq_t fq_shl_lazy(const fq_t &a, uint32_t s) {
  fq_t r;
  r.v[0] = a.v[0] << s;
#pragma unroll
  for (int j = 1; j < FQ_LIMBS; j++) r.v[j] = __funnelshift_l(a.v[j - 1], a.v[j], s);
  return r;
}

__device__ __forceinline__ fq_t fq_neg(const fq_t &a) { return fq_sub(fq_zero(), a); }

__device__ __forceinline__ fq_t fq_dbl(const fq_t &a) { return fq_add(a, a); }

// [0, 2q) -> [0, q)
__device__ __forceinline__ fq_t fq_canon(const fq_t &a) {
  const uint32_t q[FQ_LIMBS] = BLS_Q;
  uint32_t d[FQ_LIMBS];
  d[0] = sub_cc(a.v[0], q[0]);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS; j++) d[j] = subc_cc(a.v[j], q[j]);
  const uint32_t borrow = subc(0u, 0u);
  fq_t r;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) r.v[j] = borrow ? a.v[j] : d[j];
  return r;
}

__device__ __forceinline__ bool fq_is_zero(const fq_t &a) {
  const fq_t c = fq_canon(a);
  uint32_t acc = 0;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) acc |= c.v[j];
  return acc == 0;
}

__device__ __forceinline__ bool fq_eq(const fq_t &a, const fq_t &b) {
  const fq_t x = fq_canon(a), y = fq_canon(b);
  uint32_t acc = 0;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) acc |= x.v[j] ^ y.v[j];
  return acc == 0;
}

__device__ __forceinline__ fq_t fq_select(bool c, const fq_t &a, const fq_t &b) {
  fq_t r;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) r.v[j] = c ? a.v[j] : b.v[j];
  return r;
}

// a^(q-2) = a^-1 (0 -> 0): left-to-right 4-bit fixed windows over the exponent.
static __device__ __noinline__ fq_t fq_inv(const fq_t &a) {
  const uint32_t e[FQ_LIMBS] = BLS_QM2;
  fq_t tbl[16];
  tbl[0] = fq_one();
  tbl[1] = a;
#pragma unroll 1
  for (int i = 2; i < 16; i++) tbl[i] = fq_mul(tbl[i - 1], a);
  fq_t r = fq_one();
  bool started = false;
#pragma unroll 1
  for (int w = FQ_LIMBS * 8 - 1; w >= 0; w--) {
    const uint32_t nib = (e[w >> 3] >> ((w & 7) * 4)) & 15u;
    if (started) {
      r = fq_sqr(r);
      r = fq_sqr(r);
      r = fq_sqr(r);
      r = fq_sqr(r);
    }
    if (nib) {
      r = started ? fq_mul(r, tbl[nib]) : tbl[nib];
      started = true;
    }
  }
  return r;
}

// ---- variable-time inversion by Bernstein-Yang divsteps (fq_divstep.cuh) ----
// Montgomery-form inverse (0 -> 0).  With a = xR, the integer inverse of a times R^3 through one
// Montgomery product gives x^-1 R.  One thread; about 25 batches of 30 divsteps replace the
// ~750 serial rounds of a binary extended Euclid (k_final of a 2^12-point MSM: 97 -> 71 us).
static __device__ __noinline__ fq_t fq_inv_vartime(const fq_t &a) {
  const fq_t c = fq_canon(a);
  const uint32_t q[FQ_LIMBS] = BLS_Q;
  fq_t inv;
  ds_inverse(c.v, q, inv.v);
  const uint32_t r3[FQ_LIMBS] = BLS_R3;
  return fq_mul(inv, fq_from(r3));
}

// The integer inverse of a (not times a power of R; a != 0 modulo q) by the 32 lanes of a warp
// together, which all hold a: a value below 2^383 congruent to it, on every lane.
// Lane l < 13 holds digit l (30 bits, signed) of f and g, lane 16 + l of d and e.  Applying a batch's
// matrix is then two multiply-adds per row and lane: dividing by 2^30 moves each product's low part
// one lane down and keeps its high part, and one more carry between neighbours brings the digits back
// below 2^29 + 3; no carry runs through the digits.  d and e first take the multiple m q, |m| <= 2^29,
// that makes them divisible (q = 1 mod 2^30), so a batch adds at most q/2 to their magnitude.  At most
// 37 batches (1090 divsteps) are needed for 377 bits, about 27 on average; 32 q keeps d positive.
// k_final of a 2^12-point MSM, with the map's products shared between lanes: 57 -> 27 us against a
// quad that applied the matrices limb by limb.
static __device__ __noinline__ fq_t fq_inv_warp(const fq_t &a) {
  constexpr uint32_t full = 0xffffffffu;
  const int32_t q30[13] = {1, 337838080, 8, 47665420, 155713559, 227065576, 288944623, -159596483, 154868259, 385987205, 246178736, 293990724, 110138};
  const int32_t off30[13] = {32, 73400320, 266, 451551616, 687866593, 823647492, 656293350, 261621672, 660816987, 540430500, 361526795, 817768583, 3524424};  // 32 q
  const int lane = threadIdx.x & 31, l = lane & 15;
  const bool upper = lane >= 16;
  const fq_t c = fq_canon(a);
  int32_t qd = 0, od = 0, gd = 0;
#pragma unroll
  for (int i = 0; i < 13; i++) {
    const int w = 30 * i / 32, s = 30 * i % 32;
    const uint32_t hi = w + 1 < FQ_LIMBS ? c.v[w + 1] : 0u;
    if (l == i) {
      qd = q30[i];
      od = off30[i];
      gd = (int32_t)(__funnelshift_r(c.v[w], hi, s) & 0x3fffffffu);
    }
  }
  int32_t x = upper ? 0 : qd, y = upper ? (l == 0 ? 1 : 0) : gd;
  int delta = 1;
#pragma unroll 1
  for (int batch = 0; batch < 48; batch++) {
    int32_t u, v, qq, r;
    delta = ds_batch30(delta, (uint32_t)__shfl_sync(full, x, 0), (uint32_t)__shfl_sync(full, y, 0), u, v, qq, r);
    int64_t t1 = (int64_t)u * x + (int64_t)v * y, t2 = (int64_t)qq * x + (int64_t)r * y;
    // m = -(t mod 2^30), centred; zero for f and g, whose division is exact
    const int32_t m1 = -((int32_t)(__shfl_sync(full, (uint32_t)t1, 0, 16) << 2) >> 2);
    const int32_t m2 = -((int32_t)(__shfl_sync(full, (uint32_t)t2, 0, 16) << 2) >> 2);
    t1 += (int64_t)m1 * qd;
    t2 += (int64_t)m2 * qd;
    const int32_t lo1 = (int32_t)((uint32_t)t1 << 2) >> 2, lo2 = (int32_t)((uint32_t)t2 << 2) >> 2;
    const int32_t n1 = __shfl_down_sync(full, lo1, 1, 16) + (int32_t)((t1 + (1 << 29)) >> 30);
    const int32_t n2 = __shfl_down_sync(full, lo2, 1, 16) + (int32_t)((t2 + (1 << 29)) >> 30);
    const int32_t c1 = l < 12 ? (n1 + (1 << 29)) >> 30 : 0, c2 = l < 12 ? (n2 + (1 << 29)) >> 30 : 0;
    const int32_t p1 = __shfl_up_sync(full, c1, 1, 16), p2 = __shfl_up_sync(full, c2, 1, 16);
    x = n1 - (c1 << 30) + (l ? p1 : 0);
    y = n2 - (c2 << 30) + (l ? p2 : 0);
    if (!__any_sync(full, !upper && y != 0)) break;
  }
  // f = +-1: the inverse is +-d; digits of +-d + 32 q, then 32-bit words
  const bool neg = __shfl_sync(full, x, 0) < 0;
  const int32_t z = (neg ? -x : x) + od;
  uint32_t d[13];
  int32_t carry = 0;
#pragma unroll
  for (int i = 0; i < 13; i++) {
    const int32_t t = __shfl_sync(full, z, 16 + i) + carry;
    d[i] = (uint32_t)t & 0x3fffffffu;
    carry = t >> 30;
  }
  fq_t res;
#pragma unroll
  for (int i = 0; i < FQ_LIMBS; i++) {  // word i: bits 32 i .. 32 i + 31
    const int k = 32 * i / 30, s = 32 * i % 30;
    uint32_t w = (d[k] >> s) | (d[k + 1] << (30 - s));
    if (s > 28 && k + 2 < 13) w |= d[k + 2] << (60 - s);
    res.v[i] = w;
  }
  return res;
}

// ---- 16-byte vector loads/stores of field elements ----
__device__ __forceinline__ void fq_load(fq_t &r, const uint4 *p) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const uint4 u = p[k];
    r.v[4 * k + 0] = u.x;
    r.v[4 * k + 1] = u.y;
    r.v[4 * k + 2] = u.z;
    r.v[4 * k + 3] = u.w;
  }
}
__device__ __forceinline__ void fq_store(uint4 *p, const fq_t &a) {
#pragma unroll
  for (int k = 0; k < 3; k++) p[k] = make_uint4(a.v[4 * k], a.v[4 * k + 1], a.v[4 * k + 2], a.v[4 * k + 3]);
}

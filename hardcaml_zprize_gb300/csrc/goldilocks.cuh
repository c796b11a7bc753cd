// The Goldilocks field (p = 2^64 - 2^32 + 1) for the NTT kernels, and short transforms whose roots
// are powers of two.  The functions compile for the host too (plain C++), so their arithmetic can
// be checked without a GPU.
//
// Facts used: 2^64 = 2^32 - 1, 2^96 = -1 (mod p).  The reference's 16th root of unity is 2^156
// (zprize/ntt/host/gf.h:65-99, OMEGA[4]), so a transform of at most 16 points needs shifts only.
//
// Two forms of a value:
//   * uint64_t, any representative (canonical, below p, where it leaves the library);
//   * gl3, a signed 96-bit integer (three words, the top one small).  Sums and differences are
//     three-instruction carry chains with no correction; a whole 16-point transform runs on it and
//     is folded back to 64 bits once per output.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define GL_FN __host__ __device__ __forceinline__
#else
#define GL_FN inline
#endif

#define GL_P 0xffffffff00000001ull

struct gl3 {  // lo + hi 2^32 + e 2^64, e signed
  uint32_t lo, hi;
  int32_t e;
};

GL_FN uint64_t gl_pack(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

#ifndef __CUDA_ARCH__
// host forms: the same integers through 128-bit arithmetic
inline gl3 gl3_of(__int128 v) {
  gl3 r;
  r.lo = (uint32_t)v;
  r.hi = (uint32_t)(v >> 32);
  r.e = (int32_t)(v >> 64);
  return r;
}
inline __int128 gl3_val(const gl3 &a) {
  return (__int128)gl_pack(a.lo, a.hi) + (__int128)a.e * ((__int128)1 << 64);
}
#endif

GL_FN gl3 gl3_from(uint64_t a) {
  gl3 r;
  r.lo = (uint32_t)a;
  r.hi = (uint32_t)(a >> 32);
  r.e = 0;
  return r;
}

GL_FN gl3 gl3_add(const gl3 &a, const gl3 &b) {
#ifdef __CUDA_ARCH__
  gl3 r;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
      : "=&r"(r.lo), "=&r"(r.hi), "=&r"(r.e)
      : "r"(a.lo), "r"(a.hi), "r"(a.e), "r"(b.lo), "r"(b.hi), "r"(b.e));
  return r;
#else
  return gl3_of(gl3_val(a) + gl3_val(b));
#endif
}

GL_FN gl3 gl3_sub(const gl3 &a, const gl3 &b) {
#ifdef __CUDA_ARCH__
  gl3 r;
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=&r"(r.lo), "=&r"(r.hi), "=&r"(r.e)
      : "r"(a.lo), "r"(a.hi), "r"(a.e), "r"(b.lo), "r"(b.hi), "r"(b.e));
  return r;
#else
  return gl3_of(gl3_val(a) - gl3_val(b));
#endif
}

// (hi:lo) << s as three words, 0 < s < 32; the top one takes e << s too
GL_FN gl3 gl3_shl(const gl3 &a, uint32_t s) {
  gl3 r;
  r.lo = a.lo << s;
  r.hi = (a.hi << s) | (a.lo >> (32 - s));
  r.e = (int32_t)(((uint32_t)a.e << s) | (a.hi >> (32 - s)));
  return r;
}

// a 2^S modulo p, as a gl3 with a small top word.  With v = a 2^(S mod 32) in three words
// (v0, v1, v2 signed) and f = 2^32 (f^2 = f - 1, f^3 = -1):
//   S < 32:        v0 + v1 f + v2 (f - 1)
//   32 <= S < 64:  v0 f + v1 (f - 1) - v2
//   64 <= S < 96:  v0 (f - 1) - v1 - v2 f
// The multiples of f - 1 = 2^32 - 1 are wide multiplies (the multiply pipe is the idle one).
// Needs |a| 2^(S mod 32) < 2^95, so that v2 fits its word; the result is below 2^66 in magnitude.
template <uint32_t S>
GL_FN gl3 gl3_mul_pow2(const gl3 &a) {
  static_assert(S > 0 && S < 96 && S % 32 != 0, "shift out of range");
  const gl3 v = gl3_shl(a, S % 32);
#ifdef __CUDA_ARCH__
  const int32_t sx = v.e >> 31;
  gl3 r;
  if (S < 32) {
    asm("sub.cc.u32 %0, %3, %5;\n\tsubc.cc.u32 %1, %4, %6;\n\tsubc.u32 %2, 0, %6;\n\t"
        "add.cc.u32 %1, %1, %5;\n\taddc.u32 %2, %2, %6;"
        : "=&r"(r.lo), "=&r"(r.hi), "=&r"(r.e)
        : "r"(v.lo), "r"(v.hi), "r"(v.e), "r"(sx));
  } else if (S < 64) {
    const uint64_t u = (uint64_t)v.hi * 0xffffffffu;
    asm("add.cc.u32 %1, %4, %5;\n\taddc.u32 %2, 0, 0;\n\t"
        "sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %1, %7;\n\tsubc.u32 %2, %2, %7;"
        : "=&r"(r.lo), "=&r"(r.hi), "=&r"(r.e)
        : "r"((uint32_t)u), "r"((uint32_t)(u >> 32)), "r"(v.lo), "r"(v.e), "r"(sx));
  } else {
    const uint64_t u = (uint64_t)v.lo * 0xffffffffu;
    asm("sub.cc.u32 %0, %3, %5;\n\tsubc.cc.u32 %1, %4, %6;\n\tsubc.u32 %2, 0, %7;"
        : "=&r"(r.lo), "=&r"(r.hi), "=&r"(r.e)
        : "r"((uint32_t)u), "r"((uint32_t)(u >> 32)), "r"(v.hi), "r"(v.e), "r"(sx));
  }
  return r;
#else
  const __int128 v0 = v.lo, v1 = v.hi, v2 = v.e, f = (__int128)1 << 32;
  if (S < 32) return gl3_of(v0 + v1 * f + v2 * (f - 1));
  if (S < 64) return gl3_of(v0 * f + v1 * (f - 1) - v2);
  return gl3_of(v0 * (f - 1) - v1 - v2 * f);
#endif
}

// 2^64 <= a < 2^72 to 64 bits: e 2^64 = e (2^32 - 1), added as (e - 1) 2^32 + (2^32 - e), and a carry out
// of that sum (then below 2^41) adds 2^32 - 1 once more.  (The multiples of 2^32 - 1 as wide multiplies
// hold the issue port for four cycles each: 2^24 points 226.7 against 222.6 us.)
GL_FN uint64_t gl3_fold(const gl3 &a) {
#ifdef __CUDA_ARCH__
  uint32_t r0, r1, c;
  asm("add.cc.u32 %0, %3, %5;\n\taddc.cc.u32 %1, %4, %6;\n\taddc.u32 %2, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, %2;\n\tsubc.u32 %1, %1, 0;\n\tadd.u32 %1, %1, %2;"
      : "=&r"(r0), "=&r"(r1), "=&r"(c)
      : "r"(a.lo), "r"(a.hi), "r"(0u - (uint32_t)a.e), "r"((uint32_t)a.e - 1u));
  (void)c;
  return gl_pack(r0, r1);
#else
  const unsigned __int128 s =
      (unsigned __int128)gl_pack(a.lo, a.hi) + (uint64_t)(uint32_t)a.e * 0xffffffffu;
  return (uint64_t)s + ((s >> 64) ? 0xffffffffu : 0u);
#endif
}

// any 64-bit value to [0, p): a >= p exactly when a + 2^32 - 1 carries, and the sum is then a - p
GL_FN uint64_t gl_canon(uint64_t a) {
#ifdef __CUDA_ARCH__
  uint32_t t0, t1, c;
  asm("add.cc.u32 %0, %3, 0xffffffff;\n\taddc.cc.u32 %1, %4, 0;\n\taddc.u32 %2, 0, 0;"
      : "=&r"(t0), "=&r"(t1), "=&r"(c)
      : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)));
  return c ? gl_pack(t0, t1) : a;
#else
  return a >= GL_P ? a - GL_P : a;
#endif
}

// a b / 2^64 modulo p for any 64-bit a and b below p, canonical: one factor is kept times 2^64
// (Montgomery's form), so a table entry w 2^64 gives a w.  The 128-bit product (x3 x2 x1 x0) comes
// from four wide multiplies whose 64-bit addends carry the partial products' overflow.  Then, with
// p^-1 = 2^32 + 1 (mod 2^64), m = (x1 x0) (2^32 + 1) mod 2^64 makes the low words of m p equal
// (x1 x0), and the result is (x3 x2) - floor(m p / 2^64), plus p if that is negative.  m has the
// words (x0, h = x0 + x1, carry e), and floor(m p / 2^64) = m - h - e: four additions.
GL_FN uint64_t gl_mul(uint64_t a, uint64_t b) {
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  const uint64_t x = (uint64_t)a0 * b0;
  const uint64_t y = (uint64_t)a0 * b1 + (x >> 32);
  const uint64_t z = (uint64_t)a1 * b0 + (uint32_t)y;
  const uint64_t w = (uint64_t)a1 * b1 + (y >> 32) + (z >> 32);
#ifdef __CUDA_ARCH__
  uint32_t r0, r1, h, m;
  asm("add.cc.u32 %2, %4, %5;\n\taddc.u32 %3, %2, 0;\n\t"       // h, h + e
      "sub.cc.u32 %0, %4, %3;\n\tsubc.u32 %1, %2, 0;\n\t"       // m - h - e
      "sub.cc.u32 %0, %6, %0;\n\tsubc.cc.u32 %1, %7, %1;\n\tsubc.u32 %3, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, %3;\n\tsubc.u32 %1, %1, 0;"             // a borrow: minus 2^32 - 1
      : "=&r"(r0), "=&r"(r1), "=&r"(h), "=&r"(m)
      : "r"((uint32_t)x), "r"((uint32_t)z), "r"((uint32_t)w), "r"((uint32_t)(w >> 32)));
  (void)h;
  (void)m;
  return gl_pack(r0, r1);
#else
  const uint64_t xl = gl_pack((uint32_t)x, (uint32_t)z), m = xl + (xl << 32);
  const uint64_t q = m - (m >> 32) - (m < xl ? 1 : 0), r = w - q;
  return w < q ? r - 0xffffffffu : r;
#endif
}

// ---- transforms of 2^L points, L <= 4, natural order in and out ----
// Bounds (inputs below 2^64, and the constant below on input 0 only): a 4-point transform grows
// sums to below 2^66 and a shift product is below 2^66, so every shift's operand is below 2^67,
// its largest shift (28 bits) stays inside 96 bits, and outputs are below 2^70 in magnitude.
// Input 0 carries GL_BIAS = 64 p, which reaches every output unmultiplied (its path has roots of
// one only), so outputs are positive and gl3_fold applies.
GL_FN gl3 gl3_biased(const gl3 &a) {
  gl3 b;
  b.lo = 64u;  // 64 p = 2^70 - 2^38 + 2^6
  b.hi = 0xffffffc0u;
  b.e = 63;
  return gl3_add(a, b);
}

GL_FN void gl_dft2(gl3 &a, gl3 &b) {
  const gl3 s = gl3_add(a, b), d = gl3_sub(a, b);
  a = s;
  b = d;
}

// 4 points, root 2^48, in place and in natural order
GL_FN void gl_dft4(gl3 &x0, gl3 &x1, gl3 &x2, gl3 &x3) {
  const gl3 t0 = gl3_add(x0, x2), t1 = gl3_sub(x0, x2), t2 = gl3_add(x1, x3);
  const gl3 t3 = gl3_mul_pow2<48>(gl3_sub(x1, x3));
  x0 = gl3_add(t0, t2);
  x1 = gl3_add(t1, t3);
  x2 = gl3_sub(t0, t2);
  x3 = gl3_sub(t1, t3);
}

// the transform of 2^L values, input 0 already biased (gl3_biased) when L > 0
template <int L>
GL_FN void gl_dft(gl3 (&x)[1 << L]) {
  if constexpr (L == 1) {
    gl_dft2(x[0], x[1]);
  } else if constexpr (L == 2) {
    gl_dft4(x[0], x[1], x[2], x[3]);
  } else if constexpr (L == 3) {
    // 2 x 4: pairs (j, j + 4), times w8^j on the differences (w8 = -2^24, w8^2 = 2^48,
    // w8^3 = -2^72: the minus signs swap the difference), then 4 points over j
    gl3 a[4], b[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      a[j] = gl3_add(x[j], x[j + 4]);
      b[j] = (j & 1) ? gl3_sub(x[j + 4], x[j]) : gl3_sub(x[j], x[j + 4]);
    }
    b[1] = gl3_mul_pow2<24>(b[1]);
    b[2] = gl3_mul_pow2<48>(b[2]);
    b[3] = gl3_mul_pow2<72>(b[3]);
    gl_dft4(a[0], a[1], a[2], a[3]);
    gl_dft4(b[0], b[1], b[2], b[3]);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      x[2 * k] = a[k];
      x[2 * k + 1] = b[k];
    }
  } else if constexpr (L == 4) {
    // 4 x 4: 4 points over j1 for each j0 (j = 4 j1 + j0), times w16^(j0 k0), 4 points over j0;
    // output k0 + 4 k1.  w16 = -2^60, ^2 = -2^24, ^3 = 2^84, ^4 = 2^48, ^6 = -2^72, ^9 = 2^60; a
    // minus sign is taken by subtracting in the second transform's sums instead.
#pragma unroll
    for (int j = 0; j < 4; j++) gl_dft4(x[j], x[j + 4], x[j + 8], x[j + 12]);
    // now x[4 k0 + j0]
    x[5] = gl3_mul_pow2<60>(x[5]);    // minus
    x[6] = gl3_mul_pow2<24>(x[6]);    // minus
    x[7] = gl3_mul_pow2<84>(x[7]);
    x[9] = gl3_mul_pow2<24>(x[9]);    // minus
    x[10] = gl3_mul_pow2<48>(x[10]);
    x[11] = gl3_mul_pow2<72>(x[11]);  // minus
    x[13] = gl3_mul_pow2<84>(x[13]);
    x[14] = gl3_mul_pow2<72>(x[14]);  // minus
    x[15] = gl3_mul_pow2<60>(x[15]);
    // signs of (z0, z1, z2, z3): k0 = 0 + + + +, 1 + - - +, 2 + - + -, 3 + + - +
    gl3 y[16];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const gl3 z0 = x[4 * k], z1 = x[4 * k + 1], z2 = x[4 * k + 2], z3 = x[4 * k + 3];
      const bool n1 = k == 1 || k == 2, n2 = k == 1 || k == 3, n3 = k == 2;
      const gl3 t0 = n2 ? gl3_sub(z0, z2) : gl3_add(z0, z2);
      const gl3 t1 = n2 ? gl3_add(z0, z2) : gl3_sub(z0, z2);
      // t2 = +-z1 +- z3, t3 = +-z1 -+ z3; for k = 2 both are minus: the sums change sign instead
      const bool both = n1 && n3;
      const gl3 t2 = (n1 && !both) ? gl3_sub(z3, z1) : gl3_add(z1, z3);
      const gl3 d = (n1 && !both) ? gl3_add(z1, z3) : gl3_sub(z1, z3);
      const gl3 t3 = gl3_mul_pow2<48>(d);
      const bool m2 = both, m3 = n1;  // t2, t3 stand for their negatives
      y[k] = m2 ? gl3_sub(t0, t2) : gl3_add(t0, t2);
      y[k + 4] = m3 ? gl3_sub(t1, t3) : gl3_add(t1, t3);
      y[k + 8] = m2 ? gl3_add(t0, t2) : gl3_sub(t0, t2);
      y[k + 12] = m3 ? gl3_add(t1, t3) : gl3_sub(t1, t3);
    }
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = y[k];
  }
}

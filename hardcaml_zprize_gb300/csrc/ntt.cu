// NTT over the Goldilocks field (p = 2^64 - 2^32 + 1) on sm_103a: the GPU form of the reference's
// NTT track (zprize/ntt).  The transform is the reference's (zprize/ntt/host/reference.cpp:94-139):
// X[k] = sum_j x[j] w^(j k) with w = OMEGA[log2 n] of zprize/ntt/host/gf.h:65-99, natural order in
// and out.  The reference evaluates 2^24 points on the FPGA with the 4-step decomposition into
// 2^12-point transforms (zprize/ntt/docs/zprize_ntt_top.mld:6-31); this engine splits further, into
// passes of at most 2^8 points: one up to 2^8 points, two up to 2^12, three up to 2^24.  With
// n = a b c (c = 1 for two passes) and the input index j = (ja, jb, jc), most significant first:
//   pass 1: over ja for every column (jb, jc), times w_ab^(ka jb), to Z[ka][jb][jc];
//   pass 2: over jb for every (ka, jc), times w^(jc (ka + a kb)), in place;
//   pass 3: over jc for every (ka, kb), to X[ka + a kb + a b kc].
// One kernel template (k_ntt_pass) does every pass: a block holds eight of the short transforms
// (64 contiguous bytes of every row it reads or writes) and runs each as two rounds of at most 16
// points in registers, whose roots are powers of two (goldilocks.cuh).  Two passes run as one thread
// block cluster that hands the rows over through its blocks' shared memory (k_ntt_cluster).
// An inverse context (ntt_init_inverse) runs the same forward kernels, stores output k at place
// (n - k) mod n and multiplies by 1/n: the factor sits in a twist table, or in the store of a
// transform of one pass.
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/ntt_gb300.h"
#include "goldilocks.cuh"

namespace {

constexpr uint32_t NTT_MAX_LOG_N = 24;
constexpr uint32_t NTT_ONE_PASS = 8;   // largest log2 of a transform of one pass
// Two passes (one launch) up to here, three above: a cluster has at most eight blocks.  Measured on
// GB300 (us, two passes as two launches / three launches): 2^12 5.4 / 5.4, 2^13 6.8 / 5.4, 2^16 10.0 / 7.0.
constexpr uint32_t NTT_TWO_PASS = 12;
// log2 transforms per block of a split transform.  Eight: 64 contiguous bytes of every row.
// Measured with four / eight / sixteen (us): the passes of 2^24 points without their arithmetic
// 160 / 127 / 125, whole 335 / 248 / 258; 2^16 points 9.6 / 7.0, 2^12 points 5.5 / 5.4.
constexpr int NTT_LOG_COLS = 3;

// 2^i-th roots of unity of the reference's table (gf.h:65-99); OMEGA[i+1]^2 = OMEGA[i]
const uint64_t GL_OMEGA[33] = {
    0x0000000000000001ull, 0xffffffff00000000ull, 0x0001000000000000ull, 0xfffffffeff000001ull,
    0xefffffff00000001ull, 0x00003fffffffc000ull, 0x0000008000000000ull, 0xf80007ff08000001ull,
    0xbf79143ce60ca966ull, 0x1905d02a5c411f4eull, 0x9d8f2ad78bfed972ull, 0x0653b4801da1c8cfull,
    0xf2c35199959dfcb6ull, 0x1544ef2335d17997ull, 0xe0ee099310bba1e2ull, 0xf6b2cffe2306baacull,
    0x54df9630bf79450eull, 0xabd0a6e8aa3d8a0eull, 0x81281a7b05f9beacull, 0xfbd41c6b8caa3302ull,
    0x30ba2ecd5e93e76dull, 0xf502aef532322654ull, 0x4b2a18ade67246b5ull, 0xea9d5a1336fbc98bull,
    0x86cdcc31c307e171ull, 0x4bbaf5976ecfefd8ull, 0xed41d05b78d6e286ull, 0x10d78dd8915a171dull,
    0x59049500004a4485ull, 0xdfa8c93ba46d2666ull, 0x7e9bd009b86a0845ull, 0x400a7f755588e659ull,
    0x185629dcda58878cull};

// ---- host-side field arithmetic (set-up) ----
uint64_t h_mul(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) % GL_P); }
uint64_t h_pow(uint64_t b, uint64_t e) {
  uint64_t r = 1;
  for (; e; e >>= 1, b = h_mul(b, b))
    if (e & 1) r = h_mul(r, b);
  return r;
}
uint64_t h_inv(uint64_t a) { return h_pow(a, GL_P - 2); }  // Fermat; a != 0
uint64_t h_mont(uint64_t a) { return (uint64_t)(((unsigned __int128)a << 64) % GL_P); }  // gl_mul's table form

struct NttPass {
  const uint64_t *src;
  uint64_t *dst;
  // transform g = (gh, gl), gl its low log_gl bits: element i at src[gl in_c + gh in_h + i in_i],
  // output k at dst[gl out_c + gh out_h + k out_k]
  uint32_t log_gl, gl_mask;
  uint32_t in_c, in_h, in_i;
  uint32_t out_c, out_h, out_k;
  const uint64_t *tw1;  // the round boundary's factors w_m^(k0 u), tw1[k0 U + u]
  // twist tables (see TW_SHARED, TW_STEPS; k_ntt_cluster: tw the twist, tw_a the second pass's tw1)
  const uint64_t *tw, *tw_a;
  uint32_t t_k, t_g, t_shift;
  uint32_t o_mask;   // n - 1
  uint32_t reverse;  // output places negated modulo n (last pass of an inverse)
  uint64_t scale;    // outputs of an untwisted pass times this (0: none), the inverse's 1/n
};

// streaming accesses: a pass reads and writes every word once
GL_FN uint64_t gl_ldcs(const uint64_t *p) {
#ifdef __CUDA_ARCH__
  return __ldcs(p);
#else
  return *p;
#endif
}
GL_FN void gl_stcs(uint64_t *p, uint64_t v) {
#ifdef __CUDA_ARCH__
  __stcs(p, v);
#else
  *p = v;
#endif
}

// two words from global to shared memory, asynchronously (both on 16-byte boundaries)
GL_FN void gl_copy16(uint64_t *dst, const uint64_t *src) {
#ifdef __CUDA_ARCH__
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
#else
  dst[0] = src[0];
  dst[1] = src[1];
#endif
}

// ---- the pass kernel ----
// Transforms of m = 2^(L1 + L2) points in two rounds of short transforms (one where L2 = 0):
// element j = u + 2^L2 t,
//   round 1, unit u:  over t -> k0, times w_m^(k0 u);
//   round 2, unit k0: over u -> k1, output k = k0 + 2^L1 k1.
// Inside a round every root is a power of two (goldilocks.cuh), so a value meets one general
// product per round boundary and one per pass boundary (the twist).
//
// A block holds 2^LC transforms.  Round 1 reads global memory, round 2 writes it; between them
// values sit in shared memory, point (k0, u) of transform c at k0 PITCH + u C + c, or, for ROWS
// (transforms whose elements are contiguous: lanes run over u in round 1), k0 PITCH + c (U + 1) + u.
// With eight transforms PITCH = 8 (mod 16), so the half warps of both rounds meet sixteen banks.
//
// What bounds it (ncu and timings on GB300, 2^24 points): the arithmetic and the memory passes
// together.  Without arithmetic the three passes take 46 + 40 + 41 us (268 MB each, 87 to 100% of
// the measured copy bandwidth); with it 74 + 81 + 64 us: about 120 instructions per point and pass,
// of which the 32 x 32 wide multiplies hold the issue port for four cycles each.  The previous
// kernel (radix 8 with table roots, two passes of 2^12 points, one 147 KB block per SM) took
// 339 + 272 us: 5 general products per point and pass, and load, arithmetic and store phases that
// nothing overlapped.  Two passes of three such rounds took 188 + 136 us for the same reason.
template <int L1, int L2, int LC>
struct PassShape {
  static constexpr int LM = L1 + L2, U = 1 << L2, C = 1 << LC;
  static constexpr int PITCH = C * (U + 1);
  static constexpr int UNITS = C << (LM - (L1 > L2 && L2 ? L2 : L1));  // of the round with more
  static constexpr int THREADS = UNITS < 32 ? 32 : UNITS;
  static constexpr int TW_WORDS = (1 << LM) > C << L2 ? 1 << LM : C << L2;  // staged twist factors
  static constexpr size_t SMEM = L2 ? (size_t)8 * ((PITCH << L1) + TW_WORDS) : 0;
};

// base[uniform + lane], the first part the same on every thread of the block (a uniform base
// register), the second a 32-bit byte offset: no address arithmetic per access
GL_FN const uint64_t *at_of(const uint64_t *base, uint32_t uniform, uint32_t lane) {
  return (const uint64_t *)((const char *)(base + uniform) + (lane << 3));
}

// How a pass twists its outputs (the factor between it and the next pass).
enum : int {
  TW_NONE = 0,
  TW_SHARED,  // tw[k + (gl >> t_shift) t_g], the same for the block's transforms: staged in shared memory
  TW_STEPS,   // base (tw_a[g] tw[v t_k + gl]) times tw[(k - v) t_k + gl], the latter staged: 2^L2 a transform
};

// The block's share of the twist table, to shared memory behind the points: asynchronous copies
// that round 1 hides.  Read from global memory in the store loop instead, the factors' latency was
// exposed there (2^24 points: pass 1 84.6 us, pass 2 98.0 us, against 64.8 us without a twist).
template <int L1, int L2, int LC, int TWIST>
GL_FN void pass_stage_twist(const NttPass &ps, uint64_t *tws, uint32_t block, uint32_t tid, uint32_t threads) {
  using S = PassShape<L1, L2, LC>;
  const uint32_t gl = block * S::C & ps.gl_mask;
  if (TWIST == TW_SHARED) {
    const uint64_t *src = ps.tw + (gl >> ps.t_shift) * ps.t_g;
    for (uint32_t i = 2 * tid; i < (1u << S::LM); i += 2 * threads) gl_copy16(tws + i, src + i);
  } else if (TWIST == TW_STEPS) {
    for (uint32_t i = 2 * tid; i < (1u << (L2 + LC)); i += 2 * threads)
      gl_copy16(tws + i, ps.tw + ((i >> LC) << L1) * ps.t_k + gl + (i & (S::C - 1)));
  }
}

template <int T, int LC, int TWIST>
GL_FN void pass_store(const NttPass &ps, const uint64_t *tws, uint32_t gl, uint32_t gh, uint32_t v, uint32_t vstep,
                      uint64_t base, const gl3 (&x)[T]) {
  const uint32_t at = gl * ps.out_c + gh * ps.out_h + v * ps.out_k, step = vstep * ps.out_k;
#pragma unroll
  for (int t = 0; t < T; t++) {
    uint64_t y = gl3_fold(x[t]);
    if (TWIST == TW_SHARED) y = gl_mul(y, tws[v + t * vstep]);
    else if (TWIST == TW_STEPS) y = gl_mul(y, t ? gl_mul(base, tws[(t << LC) + (gl & ((1 << LC) - 1))]) : base);
    else if (ps.scale) y = gl_mul(y, ps.scale);
    else y = gl_canon(y);
    uint64_t *o;
    if (TWIST == TW_NONE && ps.reverse) {  // the inverse transform is the forward one read backwards
      o = ps.dst + ((0u - (at + t * step)) & ps.o_mask);
    } else {
      o = const_cast<uint64_t *>(at_of(ps.dst, t * step, at));
    }
    gl_stcs(o, y);
  }
}

// rows (not null): the block's transforms are in shared memory, transform c from rows[c (m + 1)]
template <int L1, int L2, int LC, bool ROWS, int TWIST>
GL_FN void pass_round1(const NttPass &ps, uint64_t *sm, uint32_t block, uint32_t tid, uint32_t threads,
                       const uint64_t *rows = nullptr) {
  using S = PassShape<L1, L2, LC>;
  constexpr int T = 1 << L1;
  for (uint32_t w = tid; w < ((uint32_t)S::U << LC); w += threads) {
    const uint32_t c = ROWS ? w >> L2 : w & (S::C - 1), u = ROWS ? w & (S::U - 1) : w >> LC;
    const uint32_t g = block * S::C + c, gl = g & ps.gl_mask, gh = g >> ps.log_gl;
    const uint32_t at = gl * ps.in_c + gh * ps.in_h + u * ps.in_i, step = S::U * ps.in_i;
    gl3 x[T];
#pragma unroll
    for (int t = 0; t < T; t++)
      x[t] = gl3_from(rows ? rows[c * ((1u << S::LM) + 1) + u + t * S::U] : gl_ldcs(at_of(ps.src, t * step, at)));
    x[0] = gl3_biased(x[0]);
    if (L1 > 0) gl_dft<L1>(x);
    if (L2 == 0) {
      pass_store<T, LC, TWIST>(ps, nullptr, gl, gh, 0, 1, 0, x);
    } else {
      uint64_t *s = sm + (ROWS ? c * (S::U + 1) + u : w);
#pragma unroll
      for (int k = 0; k < T; k++) {
        uint64_t y = gl3_fold(x[k]);
        if (k) y = gl_mul(y, ps.tw1[k * S::U + u]);
        s[k * S::PITCH] = y;
      }
    }
  }
}

template <int L1, int L2, int LC, bool ROWS, int TWIST>
GL_FN void pass_round2(const NttPass &ps, const uint64_t *sm, uint32_t block, uint32_t tid, uint32_t threads) {
  using S = PassShape<L1, L2, LC>;
  constexpr int T = 1 << L2;
  for (uint32_t w = tid; w < (1u << (L1 + LC)); w += threads) {
    const uint32_t c = w & (S::C - 1), k0 = w >> LC;
    const uint32_t g = block * S::C + c, gl = g & ps.gl_mask, gh = g >> ps.log_gl;
    const uint64_t *s = sm + k0 * S::PITCH + c * (ROWS ? S::U + 1 : 1);
    uint64_t base = 0;
    if (TWIST == TW_STEPS) base = gl_mul(ps.tw_a[g], ps.tw[k0 * ps.t_k + gl]);
    gl3 x[T];
#pragma unroll
    for (int t = 0; t < T; t++) x[t] = gl3_from(s[t * (ROWS ? 1 : S::C)]);
    x[0] = gl3_biased(x[0]);
    gl_dft<L2>(x);
    pass_store<T, LC, TWIST>(ps, sm + (S::PITCH << L1), gl, gh, k0, 1u << L1, base, x);
  }
}

template <int L1, int L2, int LC, bool ROWS, int TWIST>
__global__ void __launch_bounds__(PassShape<L1, L2, LC>::THREADS, PassShape<L1, L2, LC>::THREADS == 128 ? 6 : 1)
    k_ntt_pass(const NttPass ps) {
  using S = PassShape<L1, L2, LC>;
  extern __shared__ __align__(16) uint64_t sm[];
  if constexpr (L2 > 0 && TWIST != TW_NONE)
    pass_stage_twist<L1, L2, LC, TWIST>(ps, sm + (S::PITCH << L1), blockIdx.x, threadIdx.x, blockDim.x);
  // launched while the kernel ahead of it in the stream drains (see enqueue_ntt): from here on that
  // kernel's results are there, and the one behind may be set up
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  pass_round1<L1, L2, LC, ROWS, TWIST>(ps, sm, blockIdx.x, threadIdx.x, blockDim.x);
  if constexpr (L2 > 0) {
#ifdef __CUDA_ARCH__
    if (TWIST != TW_NONE) asm volatile("cp.async.wait_all;" ::: "memory");
#endif
    __syncthreads();
    pass_round2<L1, L2, LC, ROWS, TWIST>(ps, sm, blockIdx.x, threadIdx.x, blockDim.x);
  }
}

// The rounds (L1, L2) of a pass of 2^log_m points.
struct Rounds { int l1, l2; };
constexpr Rounds kRounds[NTT_ONE_PASS + 1] = {{0, 0}, {1, 0}, {2, 0}, {3, 0}, {2, 2},
                                              {3, 2}, {3, 3}, {4, 3}, {4, 4}};

// ---- two passes as one cluster ----
// n = a b with a = 2^LA, b = 2^LB points: block r of a / 8 takes the columns 8 r .. 8 r + 7 through
// pass 1 (the first b / 8 blocks do) and writes output ka of column jb, twisted, into the shared memory of
// the block that owns row ka (ka / 8); after a cluster barrier every block takes its eight rows through
// pass 2.  One launch and no trip through L2 between the passes: 2^12 points 3.8 us against 5.5 as two
// dependent launches and 14.3 as one block of 1024 threads.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int LA, int LB>
struct ClusterShape {
  using A = PassShape<kRounds[LA].l1, kRounds[LA].l2, 3>;
  using B = PassShape<kRounds[LB].l1, kRounds[LB].l2, 3>;
  static constexpr int BLOCKS = 1 << (LA - 3);
  static constexpr int THREADS = A::THREADS > B::THREADS ? A::THREADS : B::THREADS;
  static constexpr int MID_A = A::PITCH << kRounds[LA].l1, MID_B = B::PITCH << kRounds[LB].l1;
  static constexpr int MID = MID_A > MID_B ? MID_A : MID_B;
  static constexpr int PITCH = (1 << LB) + 1;
  static constexpr size_t SMEM = 8 * (size_t)(MID + 8 * PITCH);
};

template <int LA, int LB>
__global__ void __launch_bounds__(ClusterShape<LA, LB>::THREADS) k_ntt_cluster(const NttPass ps) {
  using C = ClusterShape<LA, LB>;
  constexpr Rounds ra = kRounds[LA], rb = kRounds[LB];
  extern __shared__ __align__(16) uint64_t sm[];
  uint64_t *rows = sm + C::MID;
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  cluster_arrive();  // answered below, before the first access to another block's memory
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  const bool columns = rank < (1u << (LB - 3));
  if (columns)
    pass_round1<ra.l1, ra.l2, 3, false, TW_NONE>(ps, sm, rank, threadIdx.x, blockDim.x);
  __syncthreads();
  cluster_wait();
  if (columns) {
    constexpr int T = 1 << ra.l2;
    for (uint32_t w = threadIdx.x; w < (1u << (ra.l1 + 3)); w += blockDim.x) {
      const uint32_t c = w & 7, k0 = w >> 3, jb = rank * 8 + c;
      uint64_t f[T];
      gl3 x[T];
#pragma unroll
      for (int t = 0; t < T; t++) f[t] = ps.tw[(jb << LA) + k0 + (t << ra.l1)];
#pragma unroll
      for (int t = 0; t < T; t++) x[t] = gl3_from(sm[k0 * C::A::PITCH + c + t * 8]);
      x[0] = gl3_biased(x[0]);
      gl_dft<ra.l2>(x);
#pragma unroll
      for (int t = 0; t < T; t++) {
        const uint32_t ka = k0 + (t << ra.l1);
        const uint64_t y = gl_mul(gl3_fold(x[t]), f[t]);
        uint32_t at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(at)
            : "r"((uint32_t)__cvta_generic_to_shared(rows + (ka & 7) * C::PITCH + jb)), "r"(ka >> 3));
        asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(at), "l"(y) : "memory");
      }
    }
  }
  cluster_arrive();
  cluster_wait();
  NttPass pb = ps;
  pb.tw1 = ps.tw_a;
  pass_round1<rb.l1, rb.l2, 3, true, TW_NONE>(pb, sm, rank, threadIdx.x, blockDim.x, rows);
  __syncthreads();
  pass_round2<rb.l1, rb.l2, 3, true, TW_NONE>(pb, sm, rank, threadIdx.x, blockDim.x);
}

struct PassKernel {
  void (*fn)(const NttPass);
  uint32_t threads;
  size_t smem;
  uint32_t cluster;  // blocks of a cluster (0: none)
};
template <int LM, int LC, bool ROWS, int TWIST>
PassKernel pass_kernel() {
  using S = PassShape<kRounds[LM].l1, kRounds[LM].l2, LC>;
  return {k_ntt_pass<kRounds[LM].l1, kRounds[LM].l2, LC, ROWS, TWIST>, (uint32_t)S::THREADS, S::SMEM, 0};
}
template <int LA, int LB>
PassKernel cluster_kernel() {
  using C = ClusterShape<LA, LB>;
  return {k_ntt_cluster<LA, LB>, (uint32_t)C::THREADS, C::SMEM, (uint32_t)C::BLOCKS};
}
// the whole transform as one block, or one cluster
PassKernel whole_kernel(uint32_t log_m) {
  switch (log_m) {
    case 0: return pass_kernel<0, 0, true, TW_NONE>();
    case 1: return pass_kernel<1, 0, true, TW_NONE>();
    case 2: return pass_kernel<2, 0, true, TW_NONE>();
    case 3: return pass_kernel<3, 0, true, TW_NONE>();
    case 4: return pass_kernel<4, 0, true, TW_NONE>();
    case 5: return pass_kernel<5, 0, true, TW_NONE>();
    case 6: return pass_kernel<6, 0, true, TW_NONE>();
    case 7: return pass_kernel<7, 0, true, TW_NONE>();
    case 8: return pass_kernel<8, 0, true, TW_NONE>();
    case 9: return cluster_kernel<5, 4>();
    case 10: return cluster_kernel<5, 5>();
    case 11: return cluster_kernel<6, 5>();
    default: return cluster_kernel<6, 6>();
  }
}
// a pass of a split transform (2^4 to 2^8 points, at least 2^4 transforms)
template <bool ROWS, int TWIST>
PassKernel split_kernel(uint32_t log_m) {
  switch (log_m) {
    case 4: return pass_kernel<4, NTT_LOG_COLS, ROWS, TWIST>();
    case 5: return pass_kernel<5, NTT_LOG_COLS, ROWS, TWIST>();
    case 6: return pass_kernel<6, NTT_LOG_COLS, ROWS, TWIST>();
    case 7: return pass_kernel<7, NTT_LOG_COLS, ROWS, TWIST>();
    default: return pass_kernel<8, NTT_LOG_COLS, ROWS, TWIST>();
  }
}

// Table set-up: out[i] = s w^(k j) for i = (k, j), j its low log_j bits, from s and the squares
// w^(2^b) in gl_mul's table form; the entries get that form too.
struct TableSpec {
  uint64_t *out;
  uint64_t n, s;
  uint32_t log_j;
  uint64_t sq[NTT_MAX_LOG_N];
};
__global__ void __launch_bounds__(256) k_ntt_table(const TableSpec ts) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ts.n) return;
  const uint32_t j = (uint32_t)i & ((1u << ts.log_j) - 1);
  const uint32_t e = j * (uint32_t)(i >> ts.log_j);
  uint64_t r = ts.s;
#pragma unroll
  for (int b = 0; b < (int)NTT_MAX_LOG_N; b++)
    if ((e >> b) & 1u) r = gl_mul(r, ts.sq[b]);
  ts.out[i] = r;
}

constexpr uint64_t kMontSq = 0xfffffffe00000001ull;  // 2^128 modulo p
// self-test hook: element-wise a op b (0 add, 1 sub, 2 mul)
__global__ void k_gl_test(int op, const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const gl3 x = gl3_from(a[i]), y = gl3_from(b[i]);
  out[i] = gl_canon(op == 0   ? gl3_fold(gl3_biased(gl3_add(x, y)))
                    : op == 1 ? gl3_fold(gl3_biased(gl3_sub(x, y)))
                              : gl_mul(gl_mul(a[i], gl_canon(b[i])), kMontSq));
}

// Linear copy of n values in 16-byte vectors; the source may be host memory that the device
// reads through the host's page tables (Grace over NVLink-C2C).
__global__ void __launch_bounds__(256) k_ntt_copy(const uint4 *src, uint4 *dst, uint64_t nvec) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
       i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// ---- host context ----
thread_local int g_err = 0;
thread_local char g_msg[512] = "";

int fail(int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_msg, sizeof(g_msg), fmt, ap);
  va_end(ap);
  g_err = code;
  return code;
}

#define NCK(x)                                                                            \
  do {                                                                                    \
    cudaError_t e_ = (x);                                                                 \
    if (e_ != cudaSuccess) return fail(NTT_ERR_CUDA, "%s: %s", #x, cudaGetErrorString(e_)); \
  } while (0)

struct NttCtx {
  int device = 0;
  uint32_t log_n = 0;
  uint64_t n = 0;
  uint64_t *d_in = nullptr, *d_out = nullptr, *d_tmp = nullptr, *d_tab = nullptr;
  // the passes in order; the first reads the input, the last writes the output, the rest d_tmp
  struct Pass {
    PassKernel k;
    NttPass ps;
    uint32_t blocks;
  } pass[3] = {};
  int n_pass = 0;
  // the device reads pageable host memory through the host's page tables: the input vector
  // moves by a copy kernel instead of a driver copy
  bool host_direct = false;
  bool inverse = false;  // outputs in reverse order and times 1/n
  int num_sms = 0;
  cudaStream_t st = nullptr;
  cudaEvent_t ev[5] = {};
  bool timing = false;
  double last_ms[4] = {0, 0, 0, 0};
  // batches: a second input and output vector, and one stream each for uploads and downloads
  uint64_t *d_in2 = nullptr, *d_out2 = nullptr;
  cudaStream_t st_up = nullptr, st_down = nullptr;
  cudaEvent_t up_done[2] = {}, comp_done[2] = {}, down_done[2] = {};
  ~NttCtx() {
    for (uint64_t *p : {d_in, d_out, d_tmp, d_tab, d_in2, d_out2})
      if (p) cudaFree(p);
    for (cudaEvent_t e : ev)
      if (e) cudaEventDestroy(e);
    for (int k = 0; k < 2; k++)
      for (cudaEvent_t e : {up_done[k], comp_done[k], down_done[k]})
        if (e) cudaEventDestroy(e);
    for (cudaStream_t x : {st, st_up, st_down})
      if (x) cudaStreamDestroy(x);
  }
};

// The passes of a transform of cx->n points and their tables, in one allocation.
int plan_passes(NttCtx *cx) {
  const uint32_t ln = cx->log_n;
  // digits of the split, most significant first
  uint32_t d[3] = {ln, 0, 0};
  const bool fused = ln > NTT_ONE_PASS && ln <= NTT_TWO_PASS;  // two passes in one launch
  cx->n_pass = ln <= NTT_TWO_PASS ? 1 : 3;
  if (fused) {
    d[1] = ln / 2;
    d[0] = ln - d[1];
  } else if (cx->n_pass == 3) {
    // Even thirds up to 2^20.  Above, passes of 2^6 and 2^8 points, whose two rounds are of one size,
    // before those of 2^7.  Measured on GB300 (us, even thirds / so): 2^21 36.3 / 33.3, 2^22 63.2 / 59.3, 2^23
    // 119.3 / 118.7; at 2^20 20.2 against 20.7.
    d[2] = ln <= 20 ? ln / 3 : ln <= 22 ? 6 : 8;
    d[1] = ln <= 20 ? (ln - d[2]) / 2 : std::min(8u, ln - d[2] - 7);
    d[0] = ln - d[1] - d[2];
  }
  const uint32_t la = d[0], lb = d[1], lc = d[2];
  const uint64_t inv_n = cx->inverse ? h_inv(cx->n % GL_P) : 1;
  struct Table {
    uint32_t log_k, log_j, log_root;  // 2^(log_k + log_j) entries s w^(k j), w of 2^log_root points
    uint64_t s;
  };
  // round factors of each pass, then the twists
  std::vector<Table> tabs;
  for (int p = 0; p < cx->n_pass + (fused ? 1 : 0); p++)
    tabs.push_back({(uint32_t)kRounds[d[p]].l1, (uint32_t)kRounds[d[p]].l2, d[p], 1});
  if (fused) {
    tabs.push_back({lb, la, ln, inv_n});  // w^(jb ka)
  } else if (cx->n_pass == 3) {
    tabs.push_back({lb, la, la + lb, 1});  // w_ab^(jb ka)
    tabs.push_back({lb, lc, lb + lc, 1});  // w_bc^(kb jc)
    tabs.push_back({la, lc, ln, inv_n});   // w^(ka jc)
  }
  std::vector<uint64_t> off;
  uint64_t total = 0;
  for (const Table &t : tabs) {
    off.push_back(total);
    total += 1ull << (t.log_k + t.log_j);
  }
  NCK(cudaMalloc(&cx->d_tab, total * 8));
  for (size_t i = 0; i < tabs.size(); i++) {
    const Table &t = tabs[i];
    TableSpec ts{};
    ts.out = cx->d_tab + off[i];
    ts.n = 1ull << (t.log_k + t.log_j);
    ts.s = h_mont(t.s);
    ts.log_j = t.log_j;
    uint64_t w = GL_OMEGA[t.log_root];
    for (uint32_t b = 0; b < NTT_MAX_LOG_N; b++, w = h_mul(w, w)) ts.sq[b] = h_mont(w);
    k_ntt_table<<<(unsigned)((ts.n + 255) / 256), 256, 0, cx->st>>>(ts);
    NCK(cudaGetLastError());
  }
  const uint32_t a = 1u << la, b = 1u << lb, c = 1u << lc;
  for (int p = 0; p < cx->n_pass; p++) {
    NttPass &ps = cx->pass[p].ps;
    ps.o_mask = (uint32_t)(cx->n - 1);
    ps.log_gl = 31;
    ps.gl_mask = 0x7fffffffu;
    ps.tw1 = cx->d_tab + off[p];
    const bool last = p + 1 == cx->n_pass;
    ps.reverse = last && cx->inverse;
    cx->pass[p].blocks = cx->n_pass == 1 ? 1 : (uint32_t)(cx->n >> (d[p] + NTT_LOG_COLS));
    if (cx->n_pass == 1) {
      cx->pass[p].k = whole_kernel(ln);
      ps.in_i = ps.out_k = 1;
      ps.scale = cx->inverse && !fused ? h_mont(inv_n) : 0;  // in the twist table of two passes
      if (fused) {
        cx->pass[p].blocks = cx->pass[p].k.cluster;
        ps.in_c = ps.out_c = 1;
        ps.in_i = b;
        ps.out_k = a;
        ps.tw_a = cx->d_tab + off[1];
        ps.tw = cx->d_tab + off[2];
      }
    } else if (p == 0) {
      cx->pass[p].k = split_kernel<false, TW_SHARED>(la);
      ps.in_c = ps.out_c = 1;
      ps.in_i = ps.out_k = b * c;
      ps.tw = cx->d_tab + off[cx->n_pass];
      ps.t_g = a;
      ps.t_shift = lc;
    } else if (!last) {
      cx->pass[p].k = split_kernel<false, TW_STEPS>(lb);
      ps.log_gl = lc;
      ps.gl_mask = c - 1;
      ps.in_c = ps.out_c = 1;
      ps.in_h = ps.out_h = b * c;
      ps.in_i = ps.out_k = c;
      ps.tw = cx->d_tab + off[4];
      ps.tw_a = cx->d_tab + off[5];
      ps.t_k = c;
      ps.t_g = 1;
    } else {
      cx->pass[p].k = split_kernel<true, TW_NONE>(d[p]);
      ps.log_gl = la;
      ps.gl_mask = a - 1;
      ps.in_c = b * c;
      ps.in_h = c;
      ps.in_i = 1;
      ps.out_c = 1;
      ps.out_h = a;
      ps.out_k = a * b;
    }
    NCK(cudaFuncSetAttribute(cx->pass[p].k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)cx->pass[p].k.smem));
  }
  NCK(cudaStreamSynchronize(cx->st));
  return 0;
}

// The transform of cx->n points from d_src to d_dst (device memory), enqueued on st.  Every pass is
// a programmatic dependent launch: it may be set up while the kernel ahead of it in the stream
// drains, and waits for that kernel's results itself before it reads the points
// (griddepcontrol.wait).  Measured (us): 2^12 points 9.3 -> 5.3, 2^19 19.6 -> 12.7, 2^24 233.7 -> 226.5.
int enqueue_ntt(NttCtx *cx, uint64_t *d_dst, const uint64_t *d_src, cudaStream_t st, bool marks) {
  for (int p = 0; p < cx->n_pass; p++) {
    NttPass ps = cx->pass[p].ps;
    ps.src = p == 0 ? d_src : cx->d_tmp;
    ps.dst = p + 1 == cx->n_pass ? d_dst : cx->d_tmp;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cx->pass[p].k.cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cx->pass[p].blocks);
    cfg.blockDim = dim3(cx->pass[p].k.threads);
    cfg.dynamicSmemBytes = cx->pass[p].k.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = cx->pass[p].k.cluster ? 2 : 1;
    NCK(cudaLaunchKernelEx(&cfg, cx->pass[p].k.fn, (const NttPass)ps));
    if (marks && p == 0) NCK(cudaEventRecord(cx->ev[2], st));
  }
  return 0;
}

}  // namespace

extern "C" {

int ntt_last_error(char *buf, size_t len) {
  if (buf && len) {
    strncpy(buf, g_msg, len - 1);
    buf[len - 1] = 0;
  }
  return g_err;
}

}  // extern "C"

namespace {

// a context of either direction (ntt_init, ntt_init_inverse)
void *ntt_create(uint32_t log_n, bool inverse) {
  g_err = 0;
  if (log_n > NTT_MAX_LOG_N) {
    fail(NTT_ERR_ARG, "ntt_init: 2^%u points is over the maximum of 2^%u", log_n, NTT_MAX_LOG_N);
    return nullptr;
  }
  auto *cx = new NttCtx();
  cx->inverse = inverse;
  const char *dev = getenv("MSM_DEVICE");
  cx->device = dev ? atoi(dev) : 0;
  cx->log_n = log_n;
  cx->n = 1ull << log_n;
  int rc = 0;
  auto step = [&](cudaError_t e, const char *what) {
    if (!rc && e != cudaSuccess) rc = fail(NTT_ERR_CUDA, "ntt_init: %s: %s", what, cudaGetErrorString(e));
  };
  step(cudaSetDevice(cx->device), "cudaSetDevice");
  int pageable = 0, host_tables = 0;
  step(cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, cx->device), "attribute");
  step(cudaDeviceGetAttribute(&host_tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables,
                              cx->device), "attribute");
  step(cudaDeviceGetAttribute(&cx->num_sms, cudaDevAttrMultiProcessorCount, cx->device), "attribute");
  const char *hd = getenv("NTT_HOST_DIRECT");
  cx->host_direct = pageable && host_tables && !(hd && strcmp(hd, "0") == 0);
  step(cudaStreamCreateWithFlags(&cx->st, cudaStreamNonBlocking), "stream");
  for (auto &e : cx->ev) step(cudaEventCreate(&e), "event");
  step(cudaMalloc(&cx->d_in, cx->n * 8), "input buffer");
  step(cudaMalloc(&cx->d_out, cx->n * 8), "output buffer");
  if (log_n > NTT_TWO_PASS) step(cudaMalloc(&cx->d_tmp, cx->n * 8), "intermediate buffer");
  if (!rc) rc = plan_passes(cx);
  if (rc) {
    delete cx;
    return nullptr;
  }
  return cx;
}

}  // namespace

extern "C" {

void *ntt_init(uint32_t log_n) { return ntt_create(log_n, false); }

void *ntt_init_inverse(uint32_t log_n) { return ntt_create(log_n, true); }

void ntt_free(void *context) { delete (NttCtx *)context; }

uint64_t ntt_input_vector_size(void *context) {
  return context ? ((NttCtx *)context)->n : 0;
}

int ntt_evaluate_device(void *context, uint64_t *d_out, const uint64_t *d_in, void *stream) {
  g_err = 0;
  auto *cx = (NttCtx *)context;
  if (!cx || !d_out || !d_in) return fail(NTT_ERR_ARG, "ntt_evaluate_device: null argument");
  if (d_out == d_in && cx->log_n <= NTT_TWO_PASS)
    return fail(NTT_ERR_ARG, "ntt_evaluate_device: the transform is out of place");
  NCK(cudaSetDevice(cx->device));
  return enqueue_ntt(cx, d_out, d_in, stream ? (cudaStream_t)stream : cx->st, false);
}

// One transform host to host on the context's stream, with its stages timed or not.
static int evaluate_host(NttCtx *cx, uint64_t *out, const uint64_t *in, bool marks) {
  // A copy kernel reads the input when the device reaches pageable memory and the buffer is
  // 16-byte aligned (GB300 at 2^24: 0.67 ms against 0.77 ms for the driver's copy); otherwise the
  // driver copies it.  The output always goes back through the driver: a kernel writing into
  // pages the host has not touched yet takes a fault per page (29 ms at 2^24 against 4.9 ms).
  const bool direct = cx->host_direct && cx->n >= 2 && ((uintptr_t)in & 15) == 0;
  const uint32_t cblocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)cx->num_sms * 8, cx->n / 512));
  if (marks) NCK(cudaEventRecord(cx->ev[0], cx->st));
  if (direct) {
    k_ntt_copy<<<cblocks, 256, 0, cx->st>>>((const uint4 *)in, (uint4 *)cx->d_in, cx->n / 2);
    NCK(cudaGetLastError());
  } else {
    NCK(cudaMemcpyAsync(cx->d_in, in, cx->n * 8, cudaMemcpyHostToDevice, cx->st));
  }
  if (marks) NCK(cudaEventRecord(cx->ev[1], cx->st));
  if (int rc = enqueue_ntt(cx, cx->d_out, cx->d_in, cx->st, marks)) return rc;
  if (marks) NCK(cudaEventRecord(cx->ev[3], cx->st));
  NCK(cudaMemcpyAsync(out, cx->d_out, cx->n * 8, cudaMemcpyDeviceToHost, cx->st));
  if (marks) NCK(cudaEventRecord(cx->ev[4], cx->st));
  NCK(cudaStreamSynchronize(cx->st));
  return 0;
}

int ntt_evaluate(void *context, uint64_t *out, const uint64_t *in, uint64_t len) {
  g_err = 0;
  auto *cx = (NttCtx *)context;
  if (!cx || !out || !in) return fail(NTT_ERR_ARG, "ntt_evaluate: null argument");
  if (len != cx->n)
    return fail(NTT_ERR_ARG, "ntt_evaluate: %llu values for a transform of %llu points",
                (unsigned long long)len, (unsigned long long)cx->n);
  NCK(cudaSetDevice(cx->device));
  if (int rc = evaluate_host(cx, out, in, true)) return rc;
  float ms[4] = {0, 0, 0, 0};
  for (int k = 0; k < 4; k++) cudaEventElapsedTime(&ms[k], cx->ev[k], cx->ev[k + 1]);
  for (int k = 0; k < 4; k++) cx->last_ms[k] = ms[k];
  return 0;
}

int ntt_field_selftest(int32_t op, const uint64_t *a, const uint64_t *b, uint64_t *out, uint64_t n) {
  g_err = 0;
  if (n && (!a || !b || !out)) return fail(NTT_ERR_ARG, "ntt_field_selftest: null argument");
  if (op < 0 || op > 2) return fail(NTT_ERR_ARG, "ntt_field_selftest: unknown operation %d", op);
  if (n == 0) return 0;
  const char *dev = getenv("MSM_DEVICE");
  NCK(cudaSetDevice(dev ? atoi(dev) : 0));
  uint64_t *d = nullptr;
  NCK(cudaMalloc(&d, n * 24));
  int rc = 0;
  if (cudaMemcpy(d, a, n * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(d + n, b, n * 8, cudaMemcpyHostToDevice) != cudaSuccess)
    rc = fail(NTT_ERR_CUDA, "ntt_field_selftest: upload failed");
  if (!rc) {
    k_gl_test<<<(unsigned)((n + 255) / 256), 256>>>(op, d, d + n, d + 2 * n, n);
    if (cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(out, d + 2 * n, n * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = fail(NTT_ERR_CUDA, "ntt_field_selftest: %s", cudaGetErrorString(cudaGetLastError()));
  }
  cudaFree(d);
  return rc;
}

int ntt_evaluate_batch(void *context, uint64_t *out, const uint64_t *in, uint64_t count) {
  g_err = 0;
  auto *cx = (NttCtx *)context;
  if (!cx || (count && (!out || !in))) return fail(NTT_ERR_ARG, "ntt_evaluate_batch: null argument");
  if (count == 0) return 0;
  NCK(cudaSetDevice(cx->device));
  // A few vectors one after another on one stream: the worker thread below and the hand-over between
  // three streams cost more than the overlap of few or small copies gains.  Measured on GB300 (us per
  // call, with the worker / so): one vector of 2^12 / 2^16 / 2^20 / 2^22 points 85 / 104 / 193 / 513 and 29 /
  // 36 / 126 / 426; four of 2^16 168 / 144, of 2^18 232 / 203, of 2^19 299 / 316; three of 2^20 382 / 379, of
  // 2^21 637 / 681; eight of 2^16 268 / 288.
  if (count <= (cx->log_n <= 18 ? 4u : cx->log_n <= 20 ? 3u : 1u)) {
    for (uint64_t i = 0; i < count; i++)
      if (int rc = evaluate_host(cx, out + i * cx->n, in + i * cx->n, false)) return rc;
    return 0;
  }
  if (!cx->d_in2) {  // the second buffer pair and the copy streams, on first use
    NCK(cudaMalloc(&cx->d_in2, cx->n * 8));
    NCK(cudaMalloc(&cx->d_out2, cx->n * 8));
    NCK(cudaStreamCreateWithFlags(&cx->st_up, cudaStreamNonBlocking));
    NCK(cudaStreamCreateWithFlags(&cx->st_down, cudaStreamNonBlocking));
    for (int k = 0; k < 2; k++) {
      NCK(cudaEventCreateWithFlags(&cx->up_done[k], cudaEventDisableTiming));
      NCK(cudaEventCreateWithFlags(&cx->comp_done[k], cudaEventDisableTiming));
      NCK(cudaEventCreateWithFlags(&cx->down_done[k], cudaEventDisableTiming));
    }
  }
  uint64_t *din[2] = {cx->d_in, cx->d_in2}, *dout[2] = {cx->d_out, cx->d_out2};
  const size_t bytes = cx->n * 8;
  // Uploads go through the driver; the copy kernel (NTT_BATCH_DIRECT=1) does not block this
  // thread but competes with the transform for the SMs (2^24, 8 vectors: 1.57 against 1.37 ms
  // per transform on GB300).
  const char *bd = getenv("NTT_BATCH_DIRECT");
  const bool direct_up = cx->host_direct && cx->n >= 2 && bd && strcmp(bd, "1") == 0;
  const uint32_t cblocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)cx->num_sms * 8, cx->n / 512));
  // A copy from or into pageable memory blocks its calling thread until it is done, so the
  // downloads run on a worker thread while this thread uploads and enqueues transforms.
  // Vector i uses slot i % 2.  Handshakes on the host: the worker takes vector i once its
  // transform is enqueued (and its completion event recorded); this thread enqueues the
  // transform of i + 2 only once the download of i is done, so no slot is overwritten while in
  // use and no event is recorded again before the worker has waited on it.
  std::mutex mu;
  std::condition_variable cv;
  uint64_t enqueued = 0, downloaded = 0;
  int worker_rc = 0;
  std::thread worker([&] {
    cudaSetDevice(cx->device);
    for (uint64_t i = 0; i < count; i++) {
      {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return enqueued > i || worker_rc < 0; });
        if (worker_rc < 0) return;
      }
      const int k = (int)(i & 1);
      cudaError_t e = cudaStreamWaitEvent(cx->st_down, cx->comp_done[k], 0);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(out + i * cx->n, dout[k], bytes, cudaMemcpyDeviceToHost, cx->st_down);
      if (e == cudaSuccess) e = cudaStreamSynchronize(cx->st_down);
      std::lock_guard<std::mutex> lk(mu);
      if (e != cudaSuccess) {
        worker_rc = -1;
        cv.notify_all();
        return;
      }
      downloaded = i + 1;
      cv.notify_all();
    }
  });
  int rc = 0;
  for (uint64_t i = 0; i < count && !rc; i++) {
    const int k = (int)(i & 1);
    if (i >= 2) {  // the download of i - 2 has emptied the output slot
      std::unique_lock<std::mutex> lk(mu);
      cv.wait(lk, [&] { return downloaded >= i - 1 || worker_rc < 0; });
      if (worker_rc < 0) break;
    }
    cudaError_t e = cudaSuccess;
    if (i >= 2) e = cudaStreamWaitEvent(cx->st_up, cx->comp_done[k], 0);  // the input slot is free
    if (e == cudaSuccess) {
      const uint64_t *src = in + i * cx->n;
      if (direct_up && ((uintptr_t)src & 15) == 0) {  // asynchronous: this thread does not block
        k_ntt_copy<<<cblocks, 256, 0, cx->st_up>>>((const uint4 *)src, (uint4 *)din[k], cx->n / 2);
        e = cudaGetLastError();
      } else {
        e = cudaMemcpyAsync(din[k], src, bytes, cudaMemcpyHostToDevice, cx->st_up);
      }
    }
    if (e == cudaSuccess) e = cudaEventRecord(cx->up_done[k], cx->st_up);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(cx->st, cx->up_done[k], 0);
    if (e != cudaSuccess) {
      rc = fail(NTT_ERR_CUDA, "ntt_evaluate_batch: %s", cudaGetErrorString(e));
      break;
    }
    if ((rc = enqueue_ntt(cx, dout[k], din[k], cx->st, false))) break;
    if ((e = cudaEventRecord(cx->comp_done[k], cx->st)) != cudaSuccess) {
      rc = fail(NTT_ERR_CUDA, "ntt_evaluate_batch: %s", cudaGetErrorString(e));
      break;
    }
    std::lock_guard<std::mutex> lk(mu);
    enqueued = i + 1;
    cv.notify_all();
  }
  if (rc) {
    std::lock_guard<std::mutex> lk(mu);
    worker_rc = -1;
    cv.notify_all();
  }
  worker.join();
  if (!rc && worker_rc < 0) rc = fail(NTT_ERR_CUDA, "ntt_evaluate_batch: a download failed");
  cudaStreamSynchronize(cx->st);
  return rc;
}

int ntt_last_timings(void *context, double *ms, int32_t max_stages) {
  auto *cx = (NttCtx *)context;
  if (!cx || !ms) return fail(NTT_ERR_ARG, "ntt_last_timings: null argument");
  const int k = std::min<int32_t>(max_stages, 4);
  for (int i = 0; i < k; i++) ms[i] = cx->last_ms[i];
  return k;
}

}  // extern "C"

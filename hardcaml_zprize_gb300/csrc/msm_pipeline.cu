// The MSM pipeline of one pass (one or many MSMs sharing one sort), all on the device:
//
//   1. k_count     signed c-bit digits of every scalar, histogram of (MSM, window, |digit|) keys;
//                  stages each block's entries by key range, with their ranks (and uploads host
//                  scalars); k_partition, k_place_count: the same for large passes, by a partition
//                  into key ranges and a count of each range in shared memory
//   2. k_scan_*    exclusive scans -> bucket offsets in the sorted array and task offsets
//   3. k_scatter_staged, k_place  (base index | sign) into bucket order (k_scatter: from the
//                  scalars again, one launch per key range, for passes without a stage)
//   4. k_tasks     split every bucket into runs of <= seg_len entries (load balance under skew)
//   5. k_accumulate persistent: each thread sums one run of bases into a partial bucket sum
//                  (the run's first base taken as is, then a 7-product mixed add per base);
//                  k_accumulate_quad, k_reduce1_quad: four lanes a run, small passes
//   6. k_merge     buckets split over several runs: sum of their partials (a quad or a block per
//                  bucket, by the number of runs)
//   7-8. few buckets: k_lines, k_bits, k_weigh, by rows, columns and bits of the buckets' numbers; else
//      k_reduce1   per run of buckets: running sum R and triangle sum A (pippenger.h:25-33),
//                  by the dedicated addition (8 products; the unified one where it fails)
//      k_reduce2/3 combine runs into groups, groups into window sums (k_reduce3_small: one
//                  quad per window of few groups), by quad additions of two product latencies
//   9. k_final     per MSM: Horner window combine (pippenger.h:36-45), map back to affine
//                  Weierstrass, add the bases without a twisted-Edwards image
//                  (driver.cpp:349-372), write g1_projective_t (bls12_377_g1.h:427-439, 667-690)
//
// Every launch has a shape fixed by the host plan; data-dependent sizes (tasks, heavy buckets)
// are read from device counters, so a pass can be captured in a CUDA graph and replayed.
#include "engine.h"
#include "curve.cuh"

#include <algorithm>

namespace {

constexpr uint32_t kAllLanes = 0xffffffffu;
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanBlock = kScanThreads * kScanItems;

// Start of every kernel of a pass.  They are programmatic dependent launches: a kernel may be set up
// while the one ahead of it in the stream drains, and waits here for that one's completion (and so
// for all before it).  pdl_begin also lets the next kernel be set up from here on; k_accumulate
// calls pdl_wait alone: its blocks hold the SMs for the whole kernel, and blocks waiting beside them
// would take the space that a server leaves for its other passes.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  asm volatile("griddepcontrol.launch_dependents;");
}

__device__ __forceinline__ void set_error(uint32_t *counters, uint32_t code, uint32_t info) {
  if (atomicCAS(&counters[CNT_ERROR], 0u, code) == 0u) counters[CNT_ERROR_INFO] = info;
}

__device__ __forceinline__ uint32_t find_job(const JobDesc *jobs, uint32_t n_jobs, uint64_t g) {
  uint32_t lo = 0, hi = n_jobs;  // last job with point_begin <= g
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].point_begin <= g) lo = mid; else hi = mid;
  }
  return lo;
}

// The scalar bits not yet consumed, least significant first, masked to 253 bits on load.
// Windows are taken in order: each take shifts the whole scalar right by c (funnel shifts in
// registers; a runtime word index into the scalar would compile to select chains).
struct ScalarBits {
  uint32_t w[8];
};

__device__ __forceinline__ ScalarBits scalar_bits(const uint4 &a, const uint4 &b) {
  ScalarBits s;
  s.w[0] = a.x; s.w[1] = a.y; s.w[2] = a.z; s.w[3] = a.w;
  s.w[4] = b.x; s.w[5] = b.y; s.w[6] = b.z; s.w[7] = b.w & 0x1fffffffu;
  return s;
}

__device__ __forceinline__ ScalarBits load_scalar(const uint4 *p) { return scalar_bits(p[0], p[1]); }

// the next c bits (1 <= c <= 31); bits past 253 read as zero
__device__ __forceinline__ uint32_t take_bits(ScalarBits &s, uint32_t c) {
  const uint32_t v = s.w[0] & ((1u << c) - 1u);
#pragma unroll
  for (int k = 0; k < 7; k++) s.w[k] = __funnelshift_r(s.w[k], s.w[k + 1], c);
  s.w[7] >>= c;
  return v;
}

// Digit of window w, the windows taken in order from 0, given the running carry
// (hardcaml/test/top/utils.ml:243-288): slice + carry; below the top window a value >= 2^(c-1)
// becomes value - 2^c with carry 1.  Returns the signed digit and updates carry.  Unsigned mode
// returns the plain slice.
__device__ __forceinline__ int32_t next_digit(ScalarBits &s, const JobDesc &jd, uint32_t w,
                                              uint32_t &carry) {
  int32_t d = (int32_t)(take_bits(s, jd.c) + carry);
  if (!jd.signed_digits) return d;
  if (w + 1 < jd.nwin && d >= (int32_t)(1u << (jd.c - 1))) {
    d -= (int32_t)(1u << jd.c);
    carry = 1;
  } else {
    carry = 0;
  }
  return d;
}

// Global bucket id of digit magnitude `mag` in window w.  Fixed-base jobs keep one bucket array
// for all windows: their entries point at the window's own table of 2^(c w) P_i instead.
__device__ __forceinline__ uint32_t bucket_key(const JobDesc &jd, uint32_t w, uint32_t mag) {
  return jd.bucket_begin + (jd.fixed ? 0u : w * jd.nb) + (mag - 1u);
}

// The part of a digit's magnitude above its window's bucket range.  Only the top window of a
// signed layout can have one: its range is capped at the largest top digit of a scalar below r,
// and a 253-bit scalar at or above r can exceed it.  That digit becomes two entries of the same
// window, nb_top and the excess (at most nb_top: the cap is at least half of 2^c_top).
__device__ __forceinline__ uint32_t top_excess(const JobDesc &jd, uint32_t w, uint32_t mag) {
  return (w + 1 == jd.nwin && mag > jd.nb_top) ? mag - jd.nb_top : 0u;
}

// the counts, counters and run-length histogram of a pass to zero
__global__ void __launch_bounds__(256) k_clear(PassBuffers pb) {
  pdl_begin();
  const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
  for (uint32_t i = i0; i < pb.n_buckets; i += n) pb.count[i] = 0;
  for (uint32_t i = i0; i < 2 * (pb.seg_len + 1); i += n) pb.len_hist[i] = 0;
  if (i0 < CNT_WORDS) pb.counters[i0] = 0;
  if (pb.bin_total)
    for (uint32_t i = i0; i < pb.n_bins; i += n) pb.bin_total[i] = 0;
}

// ---------------------------------------------------------------------------------------------
// 1. histogram
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void count_key(const PassBuffers &pb, uint32_t key, uint32_t *sh_bins) {
  if (sh_bins) atomicAdd(&sh_bins[key >> pb.bin_shift], 1u);
  if (pb.stage) return;  // the bucket counts come with the ranks in stage_digits
  // a warp whose active lanes all hit one bucket (e.g. equal scalars) adds once; otherwise
  // every lane adds on its own (distinct buckets for uniform scalars)
  const uint32_t active = __activemask();
  const int leader = __ffs(active) - 1;
  const uint32_t k0 = __shfl_sync(active, key, leader);
  if (__all_sync(active, key == k0)) {
    if ((int)(threadIdx.x & 31) == leader) atomicAdd(&pb.count[key], (uint32_t)__popc(active));
  } else {
    atomicAdd(&pb.count[key], 1u);
  }
}

// Round 1: the global bucket histogram (and, for the staged sort, the block's key-range counts).
__device__ __forceinline__ void count_digits(const PassBuffers &pb, const JobDesc &jd, ScalarBits s,
                                             uint32_t *sh_bins) {
  uint32_t carry = 0;
  for (uint32_t w = 0; w < jd.nwin; w++) {
    const int32_t d = next_digit(s, jd, w, carry);
    if (d == 0) continue;
    const uint32_t mag = (uint32_t)abs(d);
    const uint32_t extra = top_excess(jd, w, mag);
    count_key(pb, bucket_key(jd, w, mag - extra), sh_bins);
    if (extra) count_key(pb, bucket_key(jd, w, extra), sh_bins);
  }
}

// Round 2 of the staged sort: one entry into the block's chunk, at the cursor of its key range.
__device__ __forceinline__ void stage_key(const PassBuffers &pb, uint32_t key, uint32_t val, uint32_t rank,
                                          uint32_t *sh_cur, uint2 *chunk, uint32_t *ranks) {
  const uint32_t pos = atomicAdd(&sh_cur[key >> pb.bin_shift], 1u);
  if (pos < pb.stage_cap) {
    chunk[pos] = make_uint2(key, val);
    ranks[pos] = rank;
  } else {
    set_error(pb.counters, 6, pos);
  }
}

// The entries of one point, in window order, four windows per step, so that their atomics on the bucket
// counts are in flight together (a small pass is bound by their round trips: k_count of 4096 points
// 16 -> 13 us).  A bucket count's old value is the entry's rank in its bucket; one atomic per warp when its active lanes share the bucket.
__device__ __forceinline__ void stage_digits(const PassBuffers &pb, const JobDesc &jd, ScalarBits s,
                                             uint64_t bidx, uint32_t *sh_cur, uint2 *chunk,
                                             uint32_t *ranks) {
  const int lane = threadIdx.x & 31;
  uint32_t carry = 0;
  uint32_t extra_key = 0, extra_val = 0;  // a split top digit's second entry (see top_excess)
  bool extra = false;
#pragma unroll 1
  for (uint32_t w0 = 0; w0 < jd.nwin; w0 += 4) {
    uint32_t key[4], val[4], rank[4], act[4];  // act: the lanes that share the atomic, or 0
    bool ok[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t w = w0 + k;
      ok[k] = false;
      key[k] = val[k] = rank[k] = act[k] = 0;
      if (w >= jd.nwin) continue;
      const int32_t d = next_digit(s, jd, w, carry);
      if (d == 0) continue;
      const uint32_t mag = (uint32_t)abs(d);
      const uint32_t ex = top_excess(jd, w, mag);
      const uint64_t tidx = jd.tab_base + (jd.fixed ? (uint64_t)w * jd.fb_stride : 0) + bidx;
      ok[k] = true;
      key[k] = bucket_key(jd, w, mag - ex);
      val[k] = (uint32_t)tidx | (d < 0 ? 0x80000000u : 0u);
      if (ex) {
        extra = true;
        extra_key = bucket_key(jd, w, ex);
        extra_val = val[k];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (!ok[k]) continue;
      const uint32_t active = __activemask();
      const int leader = __ffs(active) - 1;
      const uint32_t k0 = __shfl_sync(active, key[k], leader);
      if (__all_sync(active, key[k] == k0)) {
        act[k] = active;
        if (lane == leader) rank[k] = atomicAdd(&pb.count[key[k]], (uint32_t)__popc(active));
      } else {
        rank[k] = atomicAdd(&pb.count[key[k]], 1u);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (act[k])
        rank[k] = __shfl_sync(act[k], rank[k], __ffs(act[k]) - 1) + __popc(act[k] & ((1u << lane) - 1u));
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (ok[k]) stage_key(pb, key[k], val[k], rank[k], sh_cur, chunk, ranks);
  }
  if (extra)
    stage_key(pb, extra_key, extra_val, atomicAdd(&pb.count[extra_key], 1u), sh_cur, chunk, ranks);
}

// One thread per point, 256 points per block.  With host_scalars set, the kernel also uploads
// the pass's scalars; with stage set, the block also writes its entries to its chunk of the
// stage, grouped by key range.
__global__ void __launch_bounds__(MSM_POINTS_PER_CHUNK) k_count(PassBuffers pb, uint64_t g_begin,
                                                                uint64_t g_end) {
  pdl_begin();
  __shared__ uint32_t sh_cur[MSM_MAX_BINS];
  const uint32_t tid = threadIdx.x;
  const bool staged = pb.stage != nullptr;
  const uint64_t g = g_begin + (uint64_t)blockIdx.x * blockDim.x + tid;
  bool ok = false;
  JobDesc jd{};
  ScalarBits s{};
  uint64_t bidx = 0;
  if (g < g_end && g < pb.n_points) {
    jd = pb.jobs[find_job(pb.jobs, pb.n_jobs, g)];
    const uint64_t i = g - jd.point_begin;
    const uint64_t si = 2 * (jd.scalar_off + i);
    uint4 a, b;
    if (pb.host_scalars) {
      // fused upload: every scalar of the pass (bases without a bucket entry included, k_final
      // reads theirs) goes from host memory to the device copy the later kernels read
      a = pb.host_scalars[si];
      b = pb.host_scalars[si + 1];
      uint4 *dst = const_cast<uint4 *>(pb.scalars) + si;
      dst[0] = a;
      dst[1] = b;
    } else {
      a = pb.scalars[si];
      b = pb.scalars[si + 1];
    }
    bidx = jd.base_off + i;
    ok = pb.flags[bidx] == BASE_OK;
    s = scalar_bits(a, b);
  }
  if (staged) {
    if (tid < MSM_MAX_BINS) sh_cur[tid] = 0;
    __syncthreads();
  }
  if (ok) count_digits(pb, jd, s, staged ? sh_cur : nullptr);
  if (!staged) return;
  __syncthreads();
  const uint64_t chunk = g_begin / MSM_POINTS_PER_CHUNK + blockIdx.x;
  if (tid == 0) {  // key-range counts -> starts (n_bins <= 32)
    uint32_t *bo = pb.blk_off + chunk * (pb.n_bins + 1);
    uint32_t acc = 0;
    for (uint32_t r = 0; r < pb.n_bins; r++) {
      const uint32_t c = sh_cur[r];
      sh_cur[r] = acc;
      bo[r] = acc;
      acc += c;
    }
    bo[pb.n_bins] = acc;
  }
  __syncthreads();
  if (ok)
    stage_digits(pb, jd, s, bidx, sh_cur, pb.stage + chunk * pb.stage_cap,
                 pb.stage_rank + chunk * pb.stage_cap);
}

// ---------------------------------------------------------------------------------------------
// 2. scans of (count, ceil(count / seg_len))
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint2 warp_incl_scan2(uint2 v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t a = __shfl_up_sync(0xffffffffu, v.x, o);
    const uint32_t b = __shfl_up_sync(0xffffffffu, v.y, o);
    if ((int)(threadIdx.x & 31) >= o) { v.x += a; v.y += b; }
  }
  return v;
}

// block-wide exclusive scan of pairs; returns this thread's exclusive prefix and the block total
__device__ __forceinline__ uint2 block_excl_scan2(uint2 v, uint2 &total) {
  __shared__ uint2 warp_tot[32];
  __shared__ uint2 tot_sh;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const uint2 inc = warp_incl_scan2(v);
  if (lane == 31) warp_tot[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const uint2 t = lane < nw ? warp_tot[lane] : make_uint2(0, 0);
    const uint2 ti = warp_incl_scan2(t);
    if (lane < nw) warp_tot[lane] = make_uint2(ti.x - t.x, ti.y - t.y);
    if (lane == 31) tot_sh = ti;
  }
  __syncthreads();
  total = tot_sh;
  const uint2 base = warp_tot[wid];
  __syncthreads();  // the shared words are reused by the next call
  return make_uint2(base.x + inc.x - v.x, base.y + inc.y - v.y);
}

__device__ __forceinline__ uint32_t ntask_of(uint32_t cnt, const PassBuffers &pb) {
  const uint32_t c = cnt + pb.seg_len - 1;
  return pb.seg_shift < 32 ? c >> pb.seg_shift : c / pb.seg_len;  // the automatic run lengths are powers of two
}

// the pass's entries and tasks, against the plan's room
__device__ __forceinline__ void scan_totals(const PassBuffers &pb, uint32_t entries, uint32_t tasks) {
  if ((uint64_t)entries > pb.max_entries) set_error(pb.counters, 1, entries);
  if (tasks > pb.max_tasks) set_error(pb.counters, 2, tasks);
  pb.counters[CNT_TASKS] = min(tasks, pb.max_tasks);
  pb.counters[CNT_ENTRIES] = entries;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(PassBuffers pb) {
  pdl_begin();
  const uint32_t base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  uint2 v = make_uint2(0, 0);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < pb.n_buckets) {
      const uint32_t c = pb.count[base + k];
      v.x += c;
      v.y += ntask_of(c, pb);
    }
  }
  uint2 total;
  block_excl_scan2(v, total);
  if (threadIdx.x == 0) {
    pb.scan_tmp[2 * blockIdx.x] = total.x;
    pb.scan_tmp[2 * blockIdx.x + 1] = total.y;
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_blocks(PassBuffers pb, uint32_t nblk) {
  pdl_begin();
  // one block: exclusive scan of the per-block totals, in chunks of kScanThreads
  __shared__ uint2 carry_sh;
  if (threadIdx.x == 0) carry_sh = make_uint2(0, 0);
  __syncthreads();
  for (uint32_t c0 = 0; c0 < nblk; c0 += kScanThreads) {
    const uint32_t i = c0 + threadIdx.x;
    const uint2 v = i < nblk ? make_uint2(pb.scan_tmp[2 * i], pb.scan_tmp[2 * i + 1]) : make_uint2(0, 0);
    uint2 total;
    const uint2 ex = block_excl_scan2(v, total);
    const uint2 cr = carry_sh;
    if (i < nblk) {
      pb.scan_tmp[2 * i] = cr.x + ex.x;
      pb.scan_tmp[2 * i + 1] = cr.y + ex.y;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry_sh = make_uint2(cr.x + total.x, cr.y + total.y);
    __syncthreads();
  }
  if (threadIdx.x == 0) scan_totals(pb, carry_sh.x, carry_sh.y);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_apply(PassBuffers pb) {
  pdl_begin();
  const uint32_t base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  uint32_t c[kScanItems];
  uint2 v = make_uint2(0, 0);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    c[k] = base + k < pb.n_buckets ? pb.count[base + k] : 0u;
    v.x += c[k];
    v.y += ntask_of(c[k], pb);
  }
  uint2 total;
  uint2 ex = block_excl_scan2(v, total);
  ex.x += pb.scan_tmp[2 * blockIdx.x];
  ex.y += pb.scan_tmp[2 * blockIdx.x + 1];
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < pb.n_buckets) {
      pb.offset[base + k] = ex.x;
      pb.taskoff[base + k] = ex.y;
    }
    ex.x += c[k];
    ex.y += ntask_of(c[k], pb);
  }
}

// The three scan kernels and k_len_hist in one, for passes of at most kScanSmallBlocks blocks of
// buckets: each block sums the counts before its own itself (at most 512 KB from L2).  A launch of
// its own costs such a pass about 4 us.
constexpr uint32_t kScanSmallBlocks = 32;

__global__ void __launch_bounds__(kScanThreads) k_scan_small(PassBuffers pb) {
  pdl_begin();
  extern __shared__ uint32_t h[];  // [seg_len + 1]
  for (uint32_t i = threadIdx.x; i <= pb.seg_len; i += blockDim.x) h[i] = 0;
  uint2 before = make_uint2(0, 0), total;
  for (uint32_t i = threadIdx.x; i < blockIdx.x * kScanBlock; i += blockDim.x) {
    const uint32_t c = pb.count[i];
    before.x += c;
    before.y += ntask_of(c, pb);
  }
  block_excl_scan2(before, before);
  const uint32_t base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  uint32_t c[kScanItems];
  uint2 v = make_uint2(0, 0);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    c[k] = base + k < pb.n_buckets ? pb.count[base + k] : 0u;
    const uint32_t nt = ntask_of(c[k], pb);
    v.x += c[k];
    v.y += nt;
    if (nt) {
      atomicAdd(&h[c[k] - (nt - 1) * pb.seg_len], 1u);
      if (nt > 1) atomicAdd(&h[pb.seg_len], nt - 1);
    }
  }
  uint2 ex = block_excl_scan2(v, total);
  ex.x += before.x;
  ex.y += before.y;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < pb.n_buckets) {
      pb.offset[base + k] = ex.x;
      if (pb.fill) pb.fill[base + k] = ex.x;  // k_scatter's slot cursor starts at the bucket's offset
      pb.taskoff[base + k] = ex.y;
    }
    ex.x += c[k];
    ex.y += ntask_of(c[k], pb);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i <= pb.seg_len; i += blockDim.x)
    if (h[i]) atomicAdd(&pb.len_hist[i], h[i]);
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) scan_totals(pb, before.x + total.x, before.y + total.y);
}

// ---------------------------------------------------------------------------------------------
// 3. scatter into bucket order, one launch per range of bucket keys [key_lo, key_hi).  A range's
//    slice of the sorted array is a few hundred MB, so its random 4-byte stores mostly merge in
//    L2 instead of each costing a DRAM read-modify-write of a whole sector; every launch
//    recomputes the digits and keeps only the entries in its range.
// ---------------------------------------------------------------------------------------------
__global__ void k_scatter(PassBuffers pb, uint32_t key_lo, uint32_t key_hi) {
  pdl_begin();
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= pb.n_points) return;
  if (pb.counters[CNT_ERROR]) return;
  const uint32_t j = find_job(pb.jobs, pb.n_jobs, g);
  const JobDesc jd = pb.jobs[j];
  const uint64_t i = g - jd.point_begin;
  const uint64_t bidx = jd.base_off + i;
  if (pb.flags[bidx] != BASE_OK) return;
  ScalarBits s = load_scalar(pb.scalars + 2 * (jd.scalar_off + i));
  const int lane = threadIdx.x & 31;
  uint32_t carry = 0;
  // four windows per step: their slot atomics are independent, so the four round trips
  // overlap instead of running one after another.  fill[key] starts at the bucket's offset in
  // the sorted array, so the atomic returns the entry's position directly.
  uint32_t extra_key = 0, extra_val = 0;  // a split top digit's second entry (see top_excess)
  bool extra = false;
#pragma unroll 1
  for (uint32_t w0 = 0; w0 < jd.nwin; w0 += 4) {
    uint32_t key[4], val[4], pos[4];
    bool ok[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t w = w0 + k;
      ok[k] = false;
      key[k] = 0;
      val[k] = 0;
      if (w < jd.nwin) {
        const int32_t d = next_digit(s, jd, w, carry);
        if (d != 0) {
          const uint32_t mag = (uint32_t)abs(d);
          const uint32_t ex = top_excess(jd, w, mag);
          key[k] = bucket_key(jd, w, mag - ex);
          ok[k] = key[k] >= key_lo && key[k] < key_hi;
          const uint64_t tidx = jd.tab_base + (jd.fixed ? (uint64_t)w * jd.fb_stride : 0) + bidx;
          val[k] = (uint32_t)tidx | (d < 0 ? 0x80000000u : 0u);
          if (ex) {
            extra_key = bucket_key(jd, w, ex);
            extra_val = val[k];
            extra = extra_key >= key_lo && extra_key < key_hi;
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      pos[k] = 0;
      if (ok[k]) {
        const uint32_t active = __activemask();
        const int leader = __ffs(active) - 1;
        const uint32_t k0 = __shfl_sync(active, key[k], leader);
        if (__all_sync(active, key[k] == k0)) {  // one bucket for the whole warp: one atomic
          uint32_t bp = 0;
          if (lane == leader) bp = atomicAdd(&pb.fill[key[k]], (uint32_t)__popc(active));
          pos[k] = __shfl_sync(active, bp, leader) + __popc(active & ((1u << lane) - 1u));
        } else {
          pos[k] = atomicAdd(&pb.fill[key[k]], 1u);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (!ok[k]) continue;
      if (pos[k] < pb.max_entries) {
        pb.vals[pos[k]] = val[k];
      } else {
        set_error(pb.counters, 3, pos[k]);
      }
    }
  }
  if (extra) {
    const uint32_t p = atomicAdd(&pb.fill[extra_key], 1u);
    if (p < pb.max_entries) {
      pb.vals[p] = extra_val;
    } else {
      set_error(pb.counters, 3, p);
    }
  }
}

// Staged sort: the entries of key range `bin`, chunk by chunk (one block per histogram block),
// each to its rank in its bucket.  The range's slice of the sorted array
// stays in L2 while the launch runs.
__global__ void __launch_bounds__(256) k_scatter_staged(PassBuffers pb, uint32_t bin, uint32_t parts) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  const uint64_t chunk = blockIdx.x / parts;
  const uint32_t *bo = pb.blk_off + chunk * (pb.n_bins + 1);
  const uint32_t lo = bo[bin], hi = min(bo[bin + 1], pb.stage_cap);
  const uint2 *st = pb.stage + chunk * pb.stage_cap;
  const uint32_t *rk = pb.stage_rank + chunk * pb.stage_cap;
  for (uint32_t e = lo + (blockIdx.x % parts) * blockDim.x + threadIdx.x; e < hi; e += parts * blockDim.x) {
    const uint2 kv = st[e];
    if (kv.x >= pb.n_buckets) {  // cannot happen for a consistent stage; never write out of bounds
      set_error(pb.counters, 7, kv.x);
      continue;
    }
    const uint32_t p = pb.offset[kv.x] + rk[e];
    if (p < pb.max_entries) pb.vals[p] = kv.y;
    else set_error(pb.counters, 3, p);
  }
}

// ---------------------------------------------------------------------------------------------
// 1 and 3 of a large pass, without an atomic or a scattered access to global memory per entry (those
// bound k_count and k_scatter_staged: two L2 round trips an entry each, 1e8 entries 3.4 ms, where the
// bytes take 0.3).  k_partition sorts the entries of a chunk of points by key range in shared memory
// and copies them out in that order; k_place_count and k_place give a key range's entries, a piece from
// every chunk, to one block (or, split by chunks, to several), which counts and ranks them in its
// shared memory.  The ranges are narrow enough that a block's slice of the sorted array stays in L2
// until its sectors are full, and a bucket's entries come in the order of the points, roughly: an order
// that is random over the whole set slows k_accumulate by 0.9% (3e6 points), by its reach in memory.
// Measured on GB300 (count + scan + scatter, ms, ranked or cursor sort / this one): 1e6 points 0.290 /
// 0.205, 2^21 without tables 0.596 / 0.415, 2^24 3.50 / 2.60, the uneven mix of 64 3.51 / 1.85, 4 x
// 50000 (3.2e6 entries) 0.112 / 0.127.  What bounds them now, in the mix: k_partition 0.55 ms (issue
// slots half used, the shared-memory pipe 65%), k_place_count 0.28 (issue slots), k_place 0.9 (L2:
// 4-byte writes, a sector each).  Sorting k_place's entries in shared memory too, to write them out in
// runs, halves the sectors and takes 1.2.
// ---------------------------------------------------------------------------------------------
constexpr int kPartThreads = 1024;

constexpr uint32_t kPlaceChunks = MSM_PLACE_CHUNKS;
constexpr uint32_t kPlaceParts = 128;  // most parts of a key range by its entries: each reads the counts of those before it
constexpr size_t kPlaceSmemMax = ((1u << MSM_MAX_PART_SHIFT) + 2 * kPlaceChunks + 1) * 4;
constexpr int kPlaceThreads = 1024;
constexpr int kPlaceUnroll = 4;

// The job of point g, walking on from job j.
__device__ __forceinline__ uint32_t next_job(const JobDesc *jobs, uint32_t n_jobs, uint32_t j, uint64_t g) {
  while (j + 1 < n_jobs && jobs[j + 1].point_begin <= g) j++;
  return j;
}

// f(key, value) for every entry of a point.  The widths that large passes use have every bit position
// known at compile time (C), with signed digits; C = 0 takes any job.
template <uint32_t C, class F>
__device__ __forceinline__ void for_digits_c(const JobDesc &jd, ScalarBits s, uint64_t bidx, F f) {
  uint32_t carry = 0;
  uint32_t tidx = (uint32_t)(jd.tab_base + bidx);  // indices are below 2^31
  const uint32_t tstep = jd.fixed ? (uint32_t)jd.fb_stride : 0u, kstep = jd.fixed ? 0u : jd.nb;
  uint32_t k0 = jd.bucket_begin - 1u;
  auto entry = [&](int32_t d, bool top) {
    if (d == 0) return;
    const uint32_t mag = (uint32_t)abs(d), ex = top && mag > jd.nb_top ? mag - jd.nb_top : 0u;
    const uint32_t val = tidx | ((uint32_t)d & 0x80000000u);
    f(k0 + mag - ex, val);
    if (ex) f(k0 + ex, val);
  };
  if constexpr (C == 0) {
    for (uint32_t w = 0; w < jd.nwin; w++) {
      entry(next_digit(s, jd, w, carry), w + 1 == jd.nwin);
      tidx += tstep;
      k0 += kstep;
    }
  } else {
    constexpr uint32_t W = (MSM_SCALAR_BITS + C - 1) / C;
#pragma unroll
    for (uint32_t w = 0; w < W; w++) {
      const uint32_t i = w * C / 32, o = w * C % 32;
      const uint32_t v = o + C <= 32 || i == 7 ? s.w[i] >> o : __funnelshift_r(s.w[i], s.w[(i + 1) & 7], o);
      int32_t d = (int32_t)((v & ((1u << C) - 1u)) + carry);
      carry = w + 1 < W && d >= (int32_t)(1u << (C - 1));
      if (carry) d -= (int32_t)(1u << C);
      entry(d, w + 1 == W);
      tidx += tstep;
      k0 += kstep;
    }
  }
}
template <class F>
__device__ __forceinline__ void for_digits(const JobDesc &jd, const ScalarBits &s, uint64_t bidx, F f) {
  if (!jd.signed_digits) return for_digits_c<0>(jd, s, bidx, f);
  switch (jd.c) {
    case 14: return for_digits_c<14>(jd, s, bidx, f);
    case 15: return for_digits_c<15>(jd, s, bidx, f);
    case 16: return for_digits_c<16>(jd, s, bidx, f);
    case 17: return for_digits_c<17>(jd, s, bidx, f);
    case 18: return for_digits_c<18>(jd, s, bidx, f);
    case 19: return for_digits_c<19>(jd, s, bidx, f);
    case 20: return for_digits_c<20>(jd, s, bidx, f);
    case 21: return for_digits_c<21>(jd, s, bidx, f);
    case 22: return for_digits_c<22>(jd, s, bidx, f);
    case 23: return for_digits_c<23>(jd, s, bidx, f);
    default: return for_digits_c<0>(jd, s, bidx, f);
  }
}

// One chunk of chunk_points points per block: its entries, grouped by key range in shared memory and
// then copied to the chunk's part of the stage (values, and keys less the range's first one).
// blk_off[range * n_chunks + chunk] is where a range starts there.
__global__ void __launch_bounds__(kPartThreads) k_partition(PassBuffers pb, uint64_t g_begin, uint64_t g_end) {
  pdl_begin();
  extern __shared__ uint32_t sh[];
  uint32_t *const cur = sh;                               // [n_bins] counts, then cursors
  uint32_t *const sval = sh + pb.n_bins;                  // [stage_cap]
  uint16_t *const skey = (uint16_t *)(sval + pb.stage_cap);  // [stage_cap]
  const uint32_t tid = threadIdx.x, low = (1u << pb.bin_shift) - 1u;
  for (uint32_t i = tid; i < pb.n_bins; i += kPartThreads) cur[i] = 0;
  const uint64_t c0 = g_begin + (uint64_t)blockIdx.x * pb.chunk_points;
  const uint64_t c1 = min(min(c0 + pb.chunk_points, g_end), pb.n_points);
  const uint64_t chunk = c0 / pb.chunk_points;
  const uint32_t j0 = find_job(pb.jobs, pb.n_jobs, c0);
  __syncthreads();
  uint32_t j = j0;
  for (uint64_t g = c0 + tid; g < c1; g += kPartThreads) {
    j = next_job(pb.jobs, pb.n_jobs, j, g);
    const JobDesc jd = pb.jobs[j];
    const uint64_t i = g - jd.point_begin;
    const uint64_t si = 2 * (jd.scalar_off + i);
    uint4 a, b;
    if (pb.host_scalars) {  // fused upload, see k_count
      a = pb.host_scalars[si];
      b = pb.host_scalars[si + 1];
      uint4 *dst = const_cast<uint4 *>(pb.scalars) + si;
      dst[0] = a;
      dst[1] = b;
    } else {
      a = pb.scalars[si];
      b = pb.scalars[si + 1];
    }
    if (pb.flags[jd.base_off + i] != BASE_OK) continue;
    for_digits(jd, scalar_bits(a, b), 0, [&](uint32_t key, uint32_t) { atomicAdd(&cur[key >> pb.bin_shift], 1u); });
  }
  __syncthreads();
  uint2 all;
  {
    const uint32_t per = (pb.n_bins + kPartThreads - 1) / kPartThreads, r0 = tid * per;
    const uint32_t r1 = min(r0 + per, pb.n_bins);
    uint2 sum = make_uint2(0, 0);
    for (uint32_t r = r0; r < r1; r++) sum.x += cur[r];
    uint32_t at = block_excl_scan2(sum, all).x;
    for (uint32_t r = r0; r < r1; r++) {
      const uint32_t c = cur[r];
      pb.blk_off[(uint64_t)r * pb.n_chunks + chunk] = at;
      if (c) atomicAdd(&pb.bin_total[r], c);
      cur[r] = at;
      at += c;
    }
    if (tid == 0) pb.blk_off[(uint64_t)pb.n_bins * pb.n_chunks + chunk] = all.x;
  }
  __syncthreads();
  j = j0;
  for (uint64_t g = c0 + tid; g < c1; g += kPartThreads) {
    j = next_job(pb.jobs, pb.n_jobs, j, g);
    const JobDesc jd = pb.jobs[j];
    const uint64_t i = g - jd.point_begin;
    const uint64_t bidx = jd.base_off + i;
    if (pb.flags[bidx] != BASE_OK) continue;
    const ScalarBits s = load_scalar(pb.scalars + 2 * (jd.scalar_off + i));
    for_digits(jd, s, bidx, [&](uint32_t key, uint32_t val) {
      const uint32_t pos = atomicAdd(&cur[key >> pb.bin_shift], 1u);
      if (pos < pb.stage_cap) {
        sval[pos] = val;
        skey[pos] = (uint16_t)(key & low);
      } else {
        set_error(pb.counters, 6, pos);
      }
    });
  }
  __syncthreads();
  const uint64_t at = chunk * pb.stage_cap;
  const uint32_t n = min(all.x, pb.stage_cap);
  for (uint32_t e = tid; e < n; e += kPartThreads) pb.stage_val[at + e] = sval[e];
  for (uint32_t e = tid; 2 * e < n; e += kPartThreads)  // the capacity is even
    ((uint32_t *)(pb.stage_key + at))[e] = ((const uint32_t *)skey)[e];
}

// A part of a key range: its entries from a stretch of the chunks.  A range of more than place_part
// entries (or more than kPlaceChunks chunks) has several parts, a block each, so that the buckets of a
// narrow top window or of repeated scalars don't leave one block with most of the work.
struct PlacePart {
  uint32_t bin, k0, nk;  // key range, its first bucket and buckets
  uint32_t part, parts;  // which of the range's parts
  uint32_t nc, total;    // chunks and entries of the part
  uint32_t *cnt, *pre, *src;
};

__device__ __forceinline__ uint32_t parts_of(const PassBuffers &pb, uint32_t total) {
  const uint32_t a = min((total + pb.place_part - 1) / pb.place_part, kPlaceParts);
  const uint32_t b = (pb.n_chunks + kPlaceChunks - 1) / kPlaceChunks;
  return min(max(max(a, b), 1u), pb.n_chunks);
}

// the part of this block; false when the block has none
__device__ __forceinline__ bool place_part(const PassBuffers &pb, uint32_t *sh, PlacePart &p) {
  __shared__ uint32_t found[3];  // range, part, parts
  const uint32_t tid = threadIdx.x;
  uint2 all;
  {
    const uint32_t per = (pb.n_bins + kPlaceThreads - 1) / kPlaceThreads, r0 = min(tid * per, pb.n_bins);
    const uint32_t r1 = min(r0 + per, pb.n_bins);
    uint2 v = make_uint2(0, 0);
    for (uint32_t r = r0; r < r1; r++) v.x += parts_of(pb, pb.bin_total[r]);
    uint32_t at = block_excl_scan2(v, all).x;
    for (uint32_t r = r0; r < r1; r++) {
      const uint32_t n = parts_of(pb, pb.bin_total[r]);
      if (blockIdx.x >= at && blockIdx.x < at + n) {
        found[0] = r;
        found[1] = blockIdx.x - at;
        found[2] = n;
      }
      at += n;
    }
  }
  if (blockIdx.x >= all.x) return false;
  __syncthreads();
  p.bin = found[0];
  p.part = found[1];
  p.parts = found[2];
  p.k0 = p.bin << pb.bin_shift;
  p.nk = min(1u << pb.bin_shift, pb.n_buckets - p.k0);
  const uint32_t c0 = (uint32_t)((uint64_t)pb.n_chunks * found[1] / p.parts);
  const uint32_t nc = (uint32_t)((uint64_t)pb.n_chunks * (found[1] + 1) / p.parts) - c0;
  p.cnt = sh;
  p.pre = sh + (1u << pb.bin_shift);
  p.src = p.pre + kPlaceChunks + 1;
  const uint32_t *row = pb.blk_off + (uint64_t)p.bin * pb.n_chunks + c0;
  const uint32_t per = (nc + kPlaceThreads - 1) / kPlaceThreads, a = min(tid * per, nc), b = min(a + per, nc);
  uint2 v = make_uint2(0, 0);
  for (uint32_t c = a; c < b; c++) {
    const uint32_t st = row[c], n = row[pb.n_chunks + c] - st;
    p.src[c] = (c0 + c) * pb.stage_cap + st;  // below 2^32: the plan's limit on entries
    p.pre[c] = n;
    v.x += n;
  }
  uint32_t at = block_excl_scan2(v, all).x;
  for (uint32_t c = a; c < b; c++) {
    const uint32_t n = p.pre[c];
    p.pre[c] = at;
    p.src[c] -= at;
    at += n;
  }
  if (tid == 0) p.pre[nc] = all.x;
  p.nc = nc;
  p.total = all.x;
  __syncthreads();
  return true;
}

// f(loaded entries, their number) for the part's entries, spread over the block's threads: its pieces, one per
// chunk, are walked as one array, the warps taking stretches of it in turn, U entries a lane in flight.
template <int U, class L, class F>
__device__ __forceinline__ void for_part_entries(const PlacePart &p, L load, F f) {
  constexpr uint32_t nw = kPlaceThreads / 32;
  const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t stretch = 256;
  uint32_t c = 0;
  for (uint32_t b0 = wid * stretch; b0 < p.total; b0 += nw * stretch) {
    uint32_t hi = p.nc;
    while (hi - c > 1) {  // the last piece that starts at or before the stretch
      const uint32_t mid = (c + hi) >> 1;
      if (p.pre[mid] <= b0) c = mid; else hi = mid;
    }
    const uint32_t b1 = min(b0 + stretch, p.total);
    uint32_t i = c, end = p.pre[c + 1], src = p.src[c], e = b0 + lane;
    auto next = [&] {
      while (e >= end) {
        i++;
        end = p.pre[i + 1];
        src = p.src[i];
      }
      return src + e;
    };
    uint2 kv[U];
    for (; e - lane + 32 * U <= b1;) {
#pragma unroll
      for (int k = 0; k < U; k++) {
        kv[k] = load(next());
        e += 32;
      }
      f(kv, U);
    }
    for (; e < b1; e += 32) {
      kv[0] = load(next());
      f(kv, 1);
    }
  }
}

// The bucket counts.  Parts of one range add theirs up; what a bucket held before is where the part's
// entries start in it.
__global__ void __launch_bounds__(kPlaceThreads, 2) k_place_count(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  extern __shared__ uint32_t sh[];
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < (1u << pb.bin_shift); i += kPlaceThreads) sh[i] = 0;
  PlacePart p;
  if (!place_part(pb, sh, p)) return;
  for_part_entries<8>(p, [&](uint32_t at) { return make_uint2(__ldcs(pb.stage_key + at), 0); },
                      [&](const uint2 *kv, int n) {
                        for (int k = 0; k < n; k++) atomicAdd(&p.cnt[kv[k].x], 1u);
                      });
  __syncthreads();
  uint32_t *const first = pb.part_first + ((uint64_t)blockIdx.x << pb.bin_shift);
  for (uint32_t k = tid; k < p.nk; k += kPlaceThreads) {
    if (p.parts == 1) {
      pb.count[p.k0 + k] = p.cnt[k];
    } else {
      first[k] = p.cnt[k];
      if (p.cnt[k]) atomicAdd(&pb.count[p.k0 + k], p.cnt[k]);
    }
  }
}

__global__ void __launch_bounds__(kPlaceThreads, 2) k_place(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  extern __shared__ uint32_t sh[];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  PlacePart p;
  if (!place_part(pb, sh, p)) return;
  const uint32_t *const first = pb.part_first + ((uint64_t)(blockIdx.x - p.part) << pb.bin_shift);
  for (uint32_t k = tid; k < p.nk; k += kPlaceThreads) {
    uint32_t at = pb.offset[p.k0 + k];
#pragma unroll 4
    for (uint32_t q = 0; q < p.part; q++) at += first[((uint64_t)q << pb.bin_shift) + k];
    p.cnt[k] = at;
  }
  __syncthreads();
  for_part_entries<kPlaceUnroll>(
      p, [&](uint32_t at) { return make_uint2(__ldcs(pb.stage_key + at), __ldcs(pb.stage_val + at)); },
      [&](const uint2 *kv, int m) {
        uint32_t pos[kPlaceUnroll];
        // one bucket for all of the warp's entries (equal scalars): one atomic
        bool same = m == kPlaceUnroll;
        if (same) {
          const uint32_t k0 = __shfl_sync(kAllLanes, kv[0].x, 0);
          for (int k = 0; k < kPlaceUnroll; k++) same = same && kv[k].x == k0;
          same = __all_sync(kAllLanes, same);
          if (same) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&p.cnt[k0], 32u * kPlaceUnroll);
            at = __shfl_sync(kAllLanes, at, 0) + lane;
            for (int k = 0; k < kPlaceUnroll; k++) pos[k] = at + 32 * k;
          }
        }
        if (!same)
          for (int k = 0; k < m; k++) pos[k] = atomicAdd(&p.cnt[kv[k].x], 1u);
        for (int k = 0; k < m; k++) {
          if (pos[k] < pb.max_entries) pb.vals[pos[k]] = kv[k].y;
          else set_error(pb.counters, 3, pos[k]);
        }
      });
}

// ---------------------------------------------------------------------------------------------
// 4. tasks: runs of <= seg_len entries, and a processing order with the longest runs first.
//    Lanes of one warp then get runs of (almost) equal length, so no lane idles while another
//    finishes a longer bucket; long runs also start first, which evens out the tail.
// ---------------------------------------------------------------------------------------------
__global__ void k_len_hist(PassBuffers pb) {
  pdl_begin();
  extern __shared__ uint32_t h[];
  for (uint32_t i = threadIdx.x; i <= pb.seg_len; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < pb.n_buckets; b += gridDim.x * blockDim.x) {
    const uint32_t cnt = pb.count[b];
    if (!cnt) continue;
    const uint32_t nt = ntask_of(cnt, pb);
    atomicAdd(&h[cnt - (nt - 1) * pb.seg_len], 1u);
    if (nt > 1) atomicAdd(&h[pb.seg_len], nt - 1);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i <= pb.seg_len; i += blockDim.x)
    if (h[i]) atomicAdd(&pb.len_hist[i], h[i]);
}

// Split buckets of at most this many runs are summed by one quad each, larger ones by a block.
constexpr uint32_t kMergeQuadMax = 16;

// One thread per bucket writes the bucket's runs and their slots in the processing order: the
// last run takes a slot in the bin of its length, the full runs of a split bucket a block of
// slots in the seg_len bin.  The block ranks its runs per bin in shared memory and reserves each
// bin's slots with one global atomic, so the few hot bin cursors (lengths cluster around the mean
// bucket load) see one atomic per block and bin.  A bin starts after the runs longer than it: every
// block sums the histogram for itself (one thread did it in a kernel of its own before).
__global__ void __launch_bounds__(256) k_tasks(PassBuffers pb) {
  pdl_begin();
  extern __shared__ uint32_t sh_bins[];  // [seg_len + 1] counts, then [seg_len + 1] slot bases
  uint32_t *bin_cnt = sh_bins, *bin_base = sh_bins + pb.seg_len + 1;
  {
    const uint32_t per = pb.seg_len / blockDim.x + 1, d0 = threadIdx.x * per;  // lengths from the longest down
    uint2 sum = make_uint2(0, 0), all;
    for (uint32_t d = d0; d < d0 + per && d <= pb.seg_len; d++) {
      bin_cnt[pb.seg_len - d] = 0;
      sum.x += pb.len_hist[pb.seg_len - d];
    }
    uint32_t at = block_excl_scan2(sum, all).x;
    for (uint32_t d = d0; d < d0 + per && d <= pb.seg_len; d++) {
      bin_base[pb.seg_len - d] = at;
      at += pb.len_hist[pb.seg_len - d];
    }
  }
  __syncthreads();
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  bool live = b < pb.n_buckets && !pb.counters[CNT_ERROR];
  uint32_t cnt = 0, nt = 0, t0 = 0, last = 0, r_last = 0, r_full = 0;
  if (live) {
    cnt = pb.count[b];
    live = cnt != 0;
  }
  if (live) {
    nt = ntask_of(cnt, pb);
    t0 = pb.taskoff[b];
    if (t0 + nt > pb.max_tasks) {
      set_error(pb.counters, 4, t0 + nt);
      live = false;
    }
  }
  if (live) {
    const uint32_t off = pb.offset[b];
    for (uint32_t k = 0; k < nt; k++) {
      Task tk;
      tk.start = off + k * pb.seg_len;
      tk.len = min(pb.seg_len, cnt - k * pb.seg_len);
      tk.bucket = b;
      tk.pad = 0;
      pb.tasks[t0 + k] = tk;
    }
    last = cnt - (nt - 1) * pb.seg_len;
    r_last = atomicAdd(&bin_cnt[last], 1u);
    if (nt > 1) {
      r_full = atomicAdd(&bin_cnt[pb.seg_len], nt - 1);
      if (nt <= kMergeQuadMax) pb.heavy[atomicAdd(&pb.counters[CNT_HEAVY], 1u)] = b;
      else pb.heavy[pb.n_buckets - 1 - atomicAdd(&pb.counters[CNT_BIG], 1u)] = b;
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i <= pb.seg_len; i += blockDim.x) {
    const uint32_t c = bin_cnt[i];
    if (c) bin_base[i] += atomicAdd(&pb.len_hist[pb.seg_len + 1 + i], c);
  }
  __syncthreads();
  if (live) {
    if (nt > 1) {
      const uint32_t base = bin_base[pb.seg_len] + r_full;
      for (uint32_t k = 0; k + 1 < nt; k++) pb.order[base + k] = t0 + k;
    }
    pb.order[bin_base[last] + r_last] = t0 + nt - 1;
  }
}

// ---------------------------------------------------------------------------------------------
// 5. bucket accumulation (persistent; warps fetch 32 tasks at a time)
// ---------------------------------------------------------------------------------------------
// The base of the current entry sits in shared memory, transposed (uint4 k of thread t at
// sh[k * 128 + t], no bank conflicts), and each operand is read right before its product.  With
// all nine words held in registers across the first three products the kernel spilled; staged,
// it fits 128 registers and runs 1.4% faster.
__device__ __forceinline__ fq_t staged_fq(const uint4 *sh, int part) {
  const uint4 a = sh[(part * 3 + 0) * 128 + threadIdx.x];
  const uint4 b = sh[(part * 3 + 1) * 128 + threadIdx.x];
  const uint4 c = sh[(part * 3 + 2) * 128 + threadIdx.x];
  fq_t r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  r.v[8] = c.x; r.v[9] = c.y; r.v[10] = c.z; r.v[11] = c.w;
  return r;
}

// te_madd with the base ((y-x)/2, (y+x)/2, d x y) read from the staging slots.  Sums and
// differences that only feed products stay unreduced (below 4q; every product is again below
// 2q), and a negative digit swaps F and G instead of negating C: with C' = -C, Z - C' = Z + C
// and Z + C' = Z - C.  The seven products are inlined: at about 400 instructions each the loop fits
// the instruction cache, and the out-of-line copy's argument moves (36 a product) are gone.  Measured
// in the mixed-add loop on GB300: 4.44e9 against 4.24e9 madd/s (the former product, 880 instructions,
// was faster out of line).
__device__ __forceinline__ xyzt_t te_madd_staged(const xyzt_t &p, const uint4 *sh, bool neg) {
  const fq_t A = fq_mul(fq_sub_lazy(p.y, p.x), staged_fq(sh, neg ? 1 : 0));
  const fq_t B = fq_mul(fq_add_lazy(p.y, p.x), staged_fq(sh, neg ? 0 : 1));
  const fq_t C = fq_mul(p.t, staged_fq(sh, 2));
  const fq_t E = fq_sub_lazy(B, A);
  const fq_t H = fq_add_lazy(B, A);
  const fq_t Zm = fq_sub_lazy(p.z, C);
  const fq_t Zp = fq_add_lazy(p.z, C);
  const fq_t F = fq_select(neg, Zp, Zm);
  const fq_t G = fq_select(neg, Zm, Zp);
  xyzt_t r;
  r.x = fq_mul(E, F);
  r.y = fq_mul(G, H);
  r.t = fq_mul(E, H);
  r.z = fq_mul(F, G);
  return r;
}

// The first entry of a run starts the sum from the base itself instead of adding it to the
// identity: x = (y+x)/2 - (y-x)/2, y = (y+x)/2 + (y-x)/2 (x negated for a negative digit), z = 1,
// t = x y -- one product instead of seven.  The warp fetches its 32 runs together, so every lane
// is at its run's first entry in the same iteration and the branch is the same on every lane.
__device__ __forceinline__ xyzt_t te_from_staged(const uint4 *sh, bool neg) {
  const fq_t ymx = staged_fq(sh, 0), ypx = staged_fq(sh, 1);
  xyzt_t r;
  r.x = neg ? fq_sub(ymx, ypx) : fq_sub(ypx, ymx);
  r.y = fq_add(ypx, ymx);
  r.z = fq_one();
  r.t = fq_mul(r.x, r.y);
  return r;
}

__global__ void __launch_bounds__(128, 4) k_accumulate(PassBuffers pb) {
  pdl_wait();
  __shared__ uint4 sh[9 * 128];
  const int lane = threadIdx.x & 31;
  const uint32_t ntasks = pb.counters[CNT_TASKS];
  if (pb.counters[CNT_ERROR]) return;
  for (;;) {
    uint32_t first = 0;
    if (lane == 0) first = atomicAdd(&pb.counters[CNT_TASK_CURSOR], 32u);
    first = __shfl_sync(0xffffffffu, first, 0);
    if (first >= ntasks) break;
    const uint32_t i = first + lane;
    if (i < ntasks) {
      const uint32_t t = pb.order[i];
      const Task tk = pb.tasks[t];
      xyzt_t acc = xyzt_identity();
      for (uint32_t e = 0; e < tk.len; e++) {
        const uint32_t v = pb.vals[tk.start + e];
        const uint32_t idx = v & 0x7fffffffu;
        if (idx >= pb.n_bases) {  // cannot happen for a consistent sort; never read out of bounds
          set_error(pb.counters, 5, idx);
          break;
        }
        const uint4 *src = pb.bases + (size_t)idx * 9;
#pragma unroll
        for (int k = 0; k < 9; k++) sh[k * 128 + threadIdx.x] = src[k];
        const bool neg = (v >> 31) != 0;
        if (e == 0) acc = te_from_staged(sh, neg);
        else acc = te_madd_staged(acc, sh, neg);
      }
      xyzt_store(pb.partials + (size_t)t * 12, acc);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// 7-8. bucket reduction: window sum = sum_b (b + 1) B_b over the window's buckets (digit
//    magnitude b + 1), the triangle sum of pippenger.h:25-33 computed in three parallel levels.
//    A run of items summarised as (R, A) -- R = sum of the items' point sums, A = sum of
//    (local position + 1) * point -- combines exactly: a run of runs has
//    A = sum_i A_i + len * sum_i i R_i, and len is a power of two (doublings only).
//    level 1: runs of 2^red_len_log2 buckets, one thread each (throughput part);
//    level 2: groups of 2^grp_len_log2 level-1 runs, one block each;
//    level 3: the groups of one window, one block per window.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t find_win(const WinDesc *wins, uint32_t n_wins, uint32_t s) {
  uint32_t lo = 0, hi = n_wins;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (wins[mid].seg_begin <= s) lo = mid; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ uint32_t find_win_grp(const WinDesc *wins, uint32_t n_wins, uint32_t g) {
  uint32_t lo = 0, hi = n_wins;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (wins[mid].grp_begin <= g) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(128) k_reduce1(PassBuffers pb) {
  pdl_begin();
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= pb.n_segs) return;
  if (pb.counters[CNT_ERROR]) return;
  const WinDesc wd = pb.wins[find_win(pb.wins, pb.n_wins, s)];
  const uint32_t L = 1u << pb.red_len_log2;
  const uint32_t lo = (s - wd.seg_begin) * L;
  const uint32_t hi = min(lo + L, wd.nb);
  xyzt_t R = xyzt_identity(), A = xyzt_identity();
  bool r_live = false, a_live = false;
  bool a_is_r = false;  // A was set to R at the first live bucket and R has not changed since
#pragma unroll 1
  for (uint32_t b = hi; b-- > lo;) {
    const uint32_t gb = wd.bucket_begin + b;
    if (pb.count[gb] != 0) {
      xyzt_t B;
      xyzt_load(B, pb.partials + (size_t)pb.taskoff[gb] * 12);
      R = r_live ? te_add_fast(R, B) : B;
      r_live = true;
      a_is_r = false;
    }
    if (r_live) {
      if (!a_live) {
        A = R;
        a_live = true;
        a_is_r = true;
      } else {
        // with A = R (an empty bucket right after the first live one) A + R is a doubling, the
        // dedicated formula's failure; a warp holding such a lane takes the unified formula for
        // this step instead of running both
        if (__any_sync(__activemask(), a_is_r)) A = te_add_ool(A, R);
        else A = te_add_fast(A, R);
        a_is_r = false;
      }
    }
  }
  xyzt_store(pb.seg_out + (size_t)s * 24, R);
  xyzt_store(pb.seg_out + (size_t)s * 24 + 12, A);
}

// ---- 4-lane cooperative point operations on distributed points ----
// Choices by lane go through fq_select, word by word: the conditional operator on a whole element
// compiles to branches that the four lanes take in turn (k_reduce2 of 2^12 points 88 against 66 us).
// The four lanes of a quad (lanes 4k..4k+3 of a warp) hold one extended point, one coordinate
// each: lane 0 X, lane 1 T, lane 2 Y, lane 3 Z.  Each lane computes one of the four independent
// products of a step and the lanes exchange what the next step needs, so a doubling costs two
// product latencies instead of eight and an addition three instead of nine, and a point takes 12
// registers per lane.  `mask` names the lanes executing the call (whole quads).
__device__ __forceinline__ int dq_lane() { return (int)(threadIdx.x & 3); }

// offset (uint4) of this lane's coordinate in an (X, Y, Z, T) record of 12 uint4
__device__ __forceinline__ int dq_off() {
  const int l = dq_lane();
  return l == 0 ? 0 : l == 1 ? 9 : l == 2 ? 3 : 6;
}
__device__ __forceinline__ fq_t dq_load(const uint4 *p) {
  fq_t r;
  fq_load(r, p + dq_off());
  return r;
}
__device__ __forceinline__ void dq_store(uint4 *p, const fq_t &v) { fq_store(p + dq_off(), v); }
__device__ __forceinline__ fq_t dq_identity() { return dq_lane() >= 2 ? fq_one() : fq_zero(); }

// the value of lane (this lane ^ x) of the quad
__device__ __forceinline__ fq_t dq_xchg(const fq_t &a, int x, uint32_t mask) {
  fq_t r;
#pragma unroll
  for (int k = 0; k < FQ_LIMBS; k++) r.v[k] = __shfl_xor_sync(mask, a.v[k], x, 4);
  return r;
}
__device__ __forceinline__ fq_t pick4(int l, const fq_t &a, const fq_t &b, const fq_t &c, const fq_t &d) {
  return fq_select(l == 0, a, fq_select(l == 1, b, fq_select(l == 2, c, d)));
}

// Sums that only feed products stay unreduced (fq_add_lazy and the like): a reduction is a chain of 25
// to 37 dependent instructions in a lone warp's latency.

// base + term (neg 0), base - term + 2q (neg ~0), or base alone (en 0); term below 2q
__device__ __forceinline__ fq_t fq_addsub(const fq_t &base, const fq_t &term, uint32_t en, uint32_t neg) {
  const uint32_t q2[FQ_LIMBS] = BLS_Q2;
  fq_t r;
  add_cc(neg, neg);  // a carry in when negating
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) r.v[j] = addc_cc(base.v[j], (term.v[j] ^ neg) & en);
  r.v[0] = add_cc(r.v[0], q2[0] & neg);
#pragma unroll
  for (int j = 1; j < FQ_LIMBS - 1; j++) r.v[j] = addc_cc(r.v[j], q2[j] & neg);
  r.v[FQ_LIMBS - 1] = addc(r.v[FQ_LIMBS - 1], q2[FQ_LIMBS - 1] & neg);
  return r;
}
// the value of lane k of the quad, on all four
__device__ __forceinline__ fq_t dq_bcast(const fq_t &a, int k, uint32_t mask) {
  fq_t r;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) r.v[j] = __shfl_sync(mask, a.v[j], k, 4);
  return r;
}

// dbl-2008-hwcd, a = -1, with 2 X Y as a product: A = X^2, B = Y^2, C = 2 Z^2, E = 2 X Y, G = B - A,
// F = G - C, H = -A - B; X3 = E F, Y3 = G H, T3 = E H, Z3 = F G.  (F and H change sign together
// here, F' = A + C - B and H' = A + B, which changes the signs of all four coordinates.)
// Products are below 1.5q, so E < 3q, G < 3.5q, F' < 6.5q, H' < 3q.
static __device__ __noinline__ fq_t dq_dbl(fq_t p, uint32_t mask) {
  const int l = dq_lane();
  const fq_t o1 = dq_xchg(p, 1, mask), o3 = dq_xchg(p, 3, mask);  // lane 1 gets X and Y
  const fq_t pr = fq_mul(fq_select(l == 1, o1, p), fq_select(l == 1, o3, p));        // A, X Y, B, Z^2 on lanes 0..3
  const fq_t A = dq_bcast(pr, 0, mask), E = fq_shl_lazy(dq_bcast(pr, 1, mask), 1);
  const fq_t B = dq_bcast(pr, 2, mask), C = fq_shl_lazy(dq_bcast(pr, 3, mask), 1);
  const fq_t H = fq_add_lazy(A, B), G = fq_sub_lazy(B, A), F = fq_sub_lazy(fq_add_lazy(A, C), B);
  return fq_mul(pick4(l, E, E, G, F), pick4(l, F, H, H, G));
}

// add-2008-hwcd-3 with k = 2d (the same formula as te_add): three product latencies
static __device__ __noinline__ fq_t dq_add_unified(fq_t p, fq_t q, uint32_t mask) {
  const uint32_t kc[FQ_LIMBS] = BLS_TE_K;
  const int l = dq_lane();
  const fq_t po = dq_xchg(p, 2, mask), qo = dq_xchg(q, 2, mask);  // lanes 0, 2 swap X and Y
  // lane 0: (Y1 - X1)(Y2 - X2) = A, lane 2: (Y1 + X1)(Y2 + X2) = B, lane 1: T1 T2, lane 3: Z1 Z2
  const fq_t m1 = l == 0 ? fq_sub(po, p) : l == 2 ? fq_add(p, po) : p;
  const fq_t m2 = l == 0 ? fq_sub(qo, q) : l == 2 ? fq_add(q, qo) : q;
  fq_t pr = fq_mul(m1, m2);
  const fq_t kpr = fq_mul(pr, fq_from(kc));
  pr = l == 1 ? kpr : l == 3 ? fq_dbl(pr) : pr;  // lane 1: C = k T1 T2, lane 3: D = 2 Z1 Z2
  // pairs {0, 2} (A, B) and {1, 3} (C, D): E = B - A, H = B + A on lanes 0, 2; F = D - C,
  // G = D + C on lanes 1, 3
  const fq_t o = dq_xchg(pr, 2, mask);
  const fq_t lo = l < 2 ? pr : o, hi = l < 2 ? o : pr;
  const fq_t u = fq_sub(hi, lo), w = fq_add(hi, lo);
  const fq_t u1 = dq_xchg(u, 1, mask);  // lane 0 gets F, lane 1 gets E
  const fq_t w3 = dq_xchg(w, 3, mask);  // lane 1 gets H, lane 2 gets G
  // X3 = E F (lane 0), T3 = E H (lane 1), Y3 = G H (lane 2), Z3 = F G (lane 3)
  return fq_mul(pick4(l, u, u1, w3, u), pick4(l, u1, w3, w, w));
}

// this lane's coordinate equals the identity's as dq_identity() writes it, on all four lanes
__device__ __forceinline__ bool dq_is_identity_bits(const fq_t &p, uint32_t mask) {
  const uint32_t one[FQ_LIMBS] = BLS_ONE;
  const bool unit = dq_lane() >= 2;  // Y and Z are one, X and T zero
  uint32_t acc = 0;
#pragma unroll
  for (int j = 0; j < FQ_LIMBS; j++) acc |= p.v[j] ^ (unit ? one[j] : 0u);
  int ok = acc == 0;
  ok &= __shfl_xor_sync(mask, ok, 1, 4);
  ok &= __shfl_xor_sync(mask, ok, 2, 4);
  return ok != 0;
}

// p + q by the dedicated formula (curve.cuh te_add_fast): two product latencies instead of three.
//   lane 0: A = (Y1 - X1)(Y2 + X2), lane 2: B = (Y1 + X1)(Y2 - X2), lane 1: C = 2 Z1 T2,
//   lane 3: D = 2 T1 Z2; then X3 = E F (lane 0), T3 = E H (1), Y3 = G H (2), Z3 = F G (3).
// Where it gives Z3 = 0 the quad takes the unified formula, or, for an operand that is the identity as
// dq_identity() writes it (padding, empty runs), the other one unchanged.  (Identity plus a point with
// X Y != 0 is right as it comes.)  Z3 = 0 modulo q leaves 0 or q, whose lowest words are 0 and 1, so one
// word tells whether to look closer.  Every lane of `mask` calls this, and the branches are uniform
// over `mask`.
static __device__ __noinline__ fq_t dq_add_rare(fq_t p, fq_t q, fq_t r, uint32_t mask) {
  const bool pid = dq_is_identity_bits(p, mask), qid = dq_is_identity_bits(q, mask);
  const int zero = fq_is_zero(r);
  const bool need = __shfl_sync(mask, zero, 3, 4) != 0 && !pid && !qid;  // Z3 = 0 on lane 3
  if (__any_sync(mask, need)) {
    const fq_t ru = dq_add_unified(p, q, mask);
    if (need) r = ru;
  }
  return pid ? q : qid ? p : r;
}

static __device__ __noinline__ fq_t dq_add(fq_t p, fq_t q, uint32_t mask) {
  const int l = dq_lane();
  const uint32_t even = (l & 1) ? 0u : ~0u, neg0 = l == 0 ? ~0u : 0u, neg2 = l == 2 ? ~0u : 0u;
  const fq_t po = dq_xchg(p, 2, mask), qo = dq_xchg(q, 2, mask);  // X <-> Y on 0, 2; T <-> Z on 1, 3
  // lane 0: Y1 - X1 and Y2 + X2, lane 2: X1 + Y1 and Y2 - X2, lanes 1, 3: the other's Z1 or T1 and T2 or Z2
  const fq_t m1 = fq_addsub(po, p, even, neg0), m2 = fq_addsub(q, qo, even, neg2);
  const fq_t pr = fq_shl_lazy(fq_mul(m1, m2), l & 1);  // A, C, B, D on lanes 0..3, below 3q
  // pairs {0, 2}: F = B - A, G = B + A; pairs {1, 3}: H = D - C, E = D + C
  const fq_t o = dq_xchg(pr, 2, mask);
  const fq_t u = fq_sub_lazy4(fq_select(l < 2, o, pr), fq_select(l < 2, pr, o)), w = fq_add_lazy(o, pr);  // below 7q, 6q
  // lane 0 lacks E, lane 2 lacks H, lane 3 lacks F and G
  const fq_t r1 = dq_xchg(fq_select(l == 1, w, u), 1, mask), r2 = dq_xchg(w, 1, mask);
  const fq_t r = fq_mul(fq_select(l == 0 || l == 3, r1, w), fq_select(l < 2, u, fq_select(l == 2, r1, r2)));
  if (__any_sync(mask, l == 3 && r.v[0] <= 1u)) return dq_add_rare(p, q, r, mask);
  return r;
}

// ---------------------------------------------------------------------------------------------
// 5-7 on quads, for passes too small to fill the GPU with one thread per run: their time is a chain
// of product latencies (about 1 us each), so a run's additions are spread over four lanes: two
// product latencies a mixed add instead of seven, two a general one instead of eight.
// A quad costs eight products' work a mixed add for a thread's seven, and 48 shuffles, so passes
// that fill the GPU keep the threads.  Measured on GB300 (one MSM, accumulate + merge, threads /
// quads, us): 4096 points 117 / 50, 16384 192 / 112, 50000 409 / 307, 2^17 724 / 760; the rules are
// kQuadEntries in the driver and kReduceQuadSegs below.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t dq_mask() { return 0xfu << (threadIdx.x & 28); }

// This lane's operand of a mixed add of base `v` (index | sign << 31): (y-x)/2 on lane 0, d x y on 1,
// (y+x)/2 on 2 (a negative digit swaps lanes 0 and 2); lane 3 multiplies Z by one.
__device__ __forceinline__ fq_t dq_load_base(const uint4 *bases, uint32_t v) {
  const int l = dq_lane();
  if (l == 3) return fq_one();
  const int part = l == 1 ? 2 : ((l == 2) != (v >> 31) ? 1 : 0);
  fq_t r;
  fq_load(r, bases + (size_t)(v & 0x7fffffffu) * 9 + part * 3);
  return r;
}

// p + base (te_madd_staged on four lanes): A = (Y-X) b0, C = T b2, B = (Y+X) b1, D = Z, then
// X3 = E F, T3 = E H, Y3 = G H, Z3 = F G.
static __device__ __noinline__ fq_t dq_madd(fq_t p, fq_t b, bool neg, uint32_t mask) {
  const int l = dq_lane();
  const uint32_t even = (l & 1) ? 0u : ~0u;
  const fq_t po = dq_xchg(p, 2, mask);
  const fq_t m1 = fq_addsub(fq_select(l & 1, p, po), p, even, l == 0 ? ~0u : 0u);
  const fq_t pr = fq_mul(m1, b);  // A, C, B, D on lanes 0..3, below 1.5q
  const fq_t o = dq_xchg(pr, 2, mask);
  const fq_t d = fq_sub_lazy(fq_select(l < 2, o, pr), fq_select(l < 2, pr, o)), a = fq_add_lazy(o, pr);
  // E, H on lanes 0, 2; F, G on 1, 3, where a negative digit negates C
  const bool swap = neg && (l & 1);
  const fq_t u = fq_select(swap, a, d), w = fq_select(swap, d, a);
  // lane 0 lacks F, lane 2 lacks G, lane 1 lacks E and H
  const fq_t r1 = dq_xchg(fq_select(l == 3, w, u), 1, mask), r2 = dq_xchg(w, 1, mask);
  return fq_mul(fq_select(l == 1, r1, fq_select(l == 2, w, u)), fq_select(l == 1, r2, fq_select(l == 3, w, r1)));
}

// the point of base v itself: X = ypx - ymx (negated for a negative digit), Y = ypx + ymx, Z = 1, T = X Y
__device__ __forceinline__ fq_t dq_from_base(const uint4 *bases, uint32_t v) {
  const int l = dq_lane();
  const uint4 *src = bases + (size_t)(v & 0x7fffffffu) * 9;
  fq_t a, b;
  fq_load(a, src);
  fq_load(b, src + 3);
  const fq_t x = (v >> 31) ? fq_sub(a, b) : fq_sub(b, a), y = fq_add(b, a);
  const fq_t t = fq_mul(x, y);
  return pick4(l, x, t, y, fq_one());
}

// One quad per run, the next base fetched while the current one is added.
__global__ void __launch_bounds__(128, 4) k_accumulate_quad(PassBuffers pb) {
  pdl_begin();
  const uint32_t ntasks = pb.counters[CNT_TASKS];
  if (pb.counters[CNT_ERROR]) return;
  const uint32_t mask = dq_mask();
  const uint32_t stride = gridDim.x * (blockDim.x / 4);
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; i < ntasks; i += stride) {
    const uint32_t t = pb.order[i];
    const Task tk = pb.tasks[t];
    uint32_t v = pb.vals[tk.start];
    if ((v & 0x7fffffffu) >= pb.n_bases) {  // cannot happen for a consistent sort; never read out of bounds
      set_error(pb.counters, 5, v & 0x7fffffffu);
      continue;
    }
    fq_t acc = dq_from_base(pb.bases, v);
    if (tk.len > 1) {
      v = pb.vals[tk.start + 1];
      bool ok = (v & 0x7fffffffu) < pb.n_bases;
      fq_t nb = ok ? dq_load_base(pb.bases, v) : fq_one();
#pragma unroll 1
      for (uint32_t e = 1; e < tk.len; e++) {
        if (!ok) {
          set_error(pb.counters, 5, v & 0x7fffffffu);
          break;
        }
        const fq_t b = nb;
        const bool neg = (v >> 31) != 0;
        if (e + 1 < tk.len) {
          v = pb.vals[tk.start + e + 1];
          ok = (v & 0x7fffffffu) < pb.n_bases;
          if (ok) nb = dq_load_base(pb.bases, v);
        }
        acc = dq_madd(acc, b, neg, mask);
      }
    }
    dq_store(pb.partials + (size_t)t * 12, acc);
  }
}

// k_reduce1 with a quad per run of buckets.  A + R right after the first live bucket, with an empty
// one between, is a doubling: it is taken as one.
__global__ void __launch_bounds__(128) k_reduce1_quad(PassBuffers pb) {
  pdl_begin();
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  if (s >= pb.n_segs) return;
  if (pb.counters[CNT_ERROR]) return;
  const uint32_t mask = dq_mask();
  const WinDesc wd = pb.wins[find_win(pb.wins, pb.n_wins, s)];
  const uint32_t L = 1u << pb.red_len_log2;
  const uint32_t lo = (s - wd.seg_begin) * L;
  const uint32_t hi = min(lo + L, wd.nb);
  fq_t R = dq_identity(), A = dq_identity();
  bool live = false, a_is_r = false;
#pragma unroll 1
  for (uint32_t b = hi; b-- > lo;) {
    const uint32_t gb = wd.bucket_begin + b;
    const bool full = pb.count[gb] != 0;
    if (full) {
      const fq_t B = dq_load(pb.partials + (size_t)pb.taskoff[gb] * 12);
      R = live ? dq_add(R, B, mask) : B;
    }
    if (full && !live) {
      A = R;
      live = a_is_r = true;
    } else if (live) {
      A = !full && a_is_r ? dq_dbl(R, mask) : dq_add(A, R, mask);
      a_is_r = false;
    }
  }
  dq_store(pb.seg_out + (size_t)s * 24, R);
  dq_store(pb.seg_out + (size_t)s * 24 + 12, A);
}

constexpr int kRedThreads = 256;
constexpr uint32_t kRedQuads = kRedThreads / 4;

// Levels 2 and 3 are chains of dependent additions, so they run on quads: every quad of the
// block executes every addition (a quad with nothing to add adds the identity), which keeps the
// warps converged for the quad shuffles.  Blocks of NT threads (NT / 4 quads): with 128 each
// SMSP runs one warp, so a step of the block's trees is shorter, but each quad sums twice as
// many items in sequence as with 256.

// Three independent sums over the block's quads at once (sh holds 3 x NT / 4 points): at each
// tree level the 3 x stride additions are spread over the quads, so the three trees take
// log2(NT / 4) + 1 rounds of dependent additions instead of 3 log2(NT / 4).  Only warps holding an
// active quad add (whole warps, so their shuffles stay converged).  The sums are valid in quad 0.
// The last warp, which most rounds leave idle, doubles its D once in every such round, up to `dbl`
// times in all (the rest after the rounds, while warp 0 goes on).
template <int NT>
__device__ __forceinline__ void block_sum3(fq_t (&X)[3], uint4 *sh, fq_t &D, uint32_t dbl) {
  constexpr uint32_t Q = NT / 4;
  const uint32_t q = threadIdx.x >> 2;
  const uint32_t warp_q0 = (threadIdx.x >> 5) * 8;  // first quad of this warp
  const bool last_warp = warp_q0 + 8 == Q;
  for (int k = 0; k < 3; k++) dq_store(sh + (k * Q + q) * 12, X[k]);
  __syncthreads();
#pragma unroll 1
  for (uint32_t stride = Q / 2; stride > 0; stride >>= 1) {
#pragma unroll 1
    for (uint32_t u0 = 0; u0 < 3 * stride; u0 += Q) {
      const uint32_t u = u0 + q;  // item u: array u / stride, element u % stride
      const bool act = u < 3 * stride;
      const uint32_t slot = act ? (u / stride) * Q + u % stride : 0;
      fq_t a = dq_identity(), o = dq_identity();
      if (act) {
        a = dq_load(sh + slot * 12);
        o = dq_load(sh + (slot + stride) * 12);
      }
      if (u0 + warp_q0 < 3 * stride) {
        a = dq_add(a, o, kAllLanes);
      } else if (last_warp && dbl) {
        D = dq_dbl(D, kAllLanes);
        dbl--;
      }
      __syncthreads();
      if (act) dq_store(sh + slot * 12, a);
      __syncthreads();
    }
  }
  if (last_warp)
    for (; dbl; dbl--) D = dq_dbl(D, kAllLanes);
  for (int k = 0; k < 3; k++) X[k] = dq_load(sh + k * Q * 12);
}

// Inclusive suffix sums over the quads: quad u gets sum_{v >= u} X_v (Hillis-Steele).
template <int NT>
__device__ __forceinline__ fq_t block_suffix_scan(fq_t X, uint4 *sh) {
  constexpr uint32_t Q = NT / 4;
  const uint32_t q = threadIdx.x >> 2;
  dq_store(sh + q * 12, X);
  __syncthreads();
#pragma unroll 1
  for (uint32_t d = 1; d < Q; d <<= 1) {
    fq_t o = dq_identity();
    if (q + d < Q) o = dq_load(sh + (q + d) * 12);
    __syncthreads();
    X = dq_add(X, o, kAllLanes);
    dq_store(sh + q * 12, X);
    __syncthreads();
  }
  return X;
}

// Combine `cnt` runs (R, A) of 2^lin_log2 buckets each into one run (A in quad 0, and R doubled
// r_dbl times in the first quad of the last warp).
// Quad u takes runs [u per, u per + per) (per a power of two) and forms SA = sum A_i,
// RR = sum R_i and T = sum (i - u per) R_i.  Then
//   A = sum_u SA_u + 2^lin_log2 (sum_u T_u + per sum_u u RR_u),  R = sum_u RR_u,
// where sum_u u RR_u = sum_{u >= 1} (suffix sum of RR at u): one block scan and three block
// sums (run together), and only quad 0 doubles.
template <int NT>
__device__ void block_combine(const uint4 *items, uint32_t cnt, uint32_t lin_log2, uint32_t r_dbl,
                              uint4 *sh, fq_t &A_out, fq_t &R_out) {
  constexpr uint32_t Q = NT / 4;
  const uint32_t q = threadIdx.x >> 2;
  uint32_t per = 1, per_log2 = 0;
  while (per * Q < cnt) {
    per <<= 1;
    per_log2++;
  }
  const uint32_t i0 = q * per;
  // the last run of the quad's share starts the sums (T = 0 R, RR = R, SA = A: no additions)
  fq_t SA = dq_identity(), T = dq_identity(), RR = dq_identity();
  if (i0 + per - 1 < cnt) {  // runs past cnt are the identity
    RR = dq_load(items + (size_t)(i0 + per - 1) * 24);
    SA = dq_load(items + (size_t)(i0 + per - 1) * 24 + 12);
  }
#pragma unroll 1
  for (uint32_t k = per - 1; k-- > 0;) {
    const uint32_t i = i0 + k;
    T = k + 2 == per ? RR : dq_add(T, RR, kAllLanes);
    fq_t R = dq_identity(), A = dq_identity();
    if (i < cnt) {
      R = dq_load(items + (size_t)i * 24);
      A = dq_load(items + (size_t)i * 24 + 12);
    }
    RR = dq_add(RR, R, kAllLanes);
    SA = dq_add(SA, A, kAllLanes);
  }
  const fq_t suf = block_suffix_scan<NT>(RR, sh);
  R_out = dq_load(sh);  // suffix at 0: the total
  __syncthreads();
  fq_t S[3] = {q ? suf : dq_identity(), T, SA};
  block_sum3<NT>(S, sh, R_out, r_dbl);
  if (q == 0) {  // lanes 0..3 of warp 0
    fq_t X = S[0];
#pragma unroll 1
    for (uint32_t k = 0; k < per_log2; k++) X = dq_dbl(X, 0xfu);
    X = dq_add(S[1], X, 0xfu);
#pragma unroll 1
    for (uint32_t k = 0; k < lin_log2; k++) X = dq_dbl(X, 0xfu);
    A_out = dq_add(X, S[2], 0xfu);
  }
}

__global__ void __launch_bounds__(kRedThreads) k_reduce2(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  const uint32_t g = blockIdx.x;
  if (g >= pb.n_grps) return;
  __shared__ uint4 sh[3 * kRedQuads * 12];
  const WinDesc wd = pb.wins[find_win_grp(pb.wins, pb.n_wins, g)];
  const uint32_t G = 1u << pb.grp_len_log2;
  const uint32_t first = (g - wd.grp_begin) * G;
  const uint32_t cnt = min(G, wd.nseg - first);
  fq_t A, R;
  // level 3 weighs the group's R by the buckets of a group, a power of two: the doublings are done
  // here, beside the sums, instead of one after another at the end of level 3
  block_combine<kRedThreads>(pb.seg_out + (size_t)(wd.seg_begin + first) * 24, cnt, pb.red_len_log2,
                    pb.red_len_log2 + pb.grp_len_log2, sh, A, R);
  if (threadIdx.x < 4) dq_store(pb.grp_out + (size_t)g * 24 + 12, A);  // one coordinate per lane
  if (threadIdx.x >= kRedThreads - 32 && threadIdx.x < kRedThreads - 28) dq_store(pb.grp_out + (size_t)g * 24, R);
}

// Windows of at most kRed3SmallMax groups (windowed MSMs: 2^(c-1) buckets make a few groups)
// are combined by one quad each, in order:
//   A = sum_i A_i + sum_i i R_i (R_i weighed by level 2),  sum_i i R_i = sum_{i >= 1} (suffix sum of R at i),
// so hundreds of windows run side by side instead of one block each.  The quads of a warp work
// on different windows, so each shuffles under its own 4-lane mask.
constexpr uint32_t kRed3SmallMax = 16;

__global__ void __launch_bounds__(128) k_reduce3_small(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;  // one window per quad
  if (gw >= pb.n_wins) return;
  const WinDesc wd = pb.wins[gw];
  const uint32_t n = wd.ngrp;
  if (n == 0 || n > kRed3SmallMax) return;
  const uint32_t mask = 0xfu << (threadIdx.x & 28);
  const uint4 *items = pb.grp_out + (size_t)wd.grp_begin * 24;
  fq_t RR = dq_load(items + (size_t)(n - 1) * 24);
  fq_t SA = dq_load(items + (size_t)(n - 1) * 24 + 12);
  fq_t T = n >= 2 ? RR : dq_identity();
#pragma unroll 1
  for (uint32_t i = n - 1; i-- > 0;) {
    const fq_t R = dq_load(items + (size_t)i * 24);
    const fq_t A = dq_load(items + (size_t)i * 24 + 12);
    SA = dq_add(SA, A, mask);
    if (i >= 1) {
      RR = dq_add(RR, R, mask);
      T = dq_add(T, RR, mask);
    }
  }
  dq_store(pb.win_sum + (size_t)gw * 12, n >= 2 ? dq_add(T, SA, mask) : SA);
}

template <int NT>
__global__ void __launch_bounds__(NT) k_reduce3(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  const uint32_t gw = blockIdx.x;
  if (gw >= pb.n_wins) return;
  __shared__ uint4 sh[3 * (NT / 4) * 12];
  const WinDesc wd = pb.wins[gw];
  if (wd.ngrp <= kRed3SmallMax) return;  // k_reduce3_small's
  fq_t A, R;
  block_combine<NT>(pb.grp_out + (size_t)wd.grp_begin * 24, wd.ngrp, 0, 0, sh, A, R);
  if (threadIdx.x < 4) dq_store(pb.win_sum + (size_t)gw * 12, A);
}

// ---------------------------------------------------------------------------------------------
// 7-8 for few buckets, by lines and bits: bucket b = hi W + lo of a window is in row hi and column lo of a
// matrix, W = 2^wl, and its weight b + 1 is W hi + (lo + 1), so with R_hi, C_lo the sums of the rows and columns
//   window sum = W sum_hi hi R_hi + sum_lo (lo + 1) C_lo,
// where a sum of i X_i is sum_k 2^k (sum of the X_i with bit k of i).  All those are plain sums, a
// block of 32 quads each (a warp per SMSP, the fastest a quad adds): k_lines the rows and columns, in
// pieces of 2^line_log2 buckets, k_bits the sums by bit (64 quads), each doubled to its weight there, side by
// side; k_weigh adds a window's up.  Two additions a bucket, as by runs, in fewer dependent ones.  Measured
// on GB300 (us, levels 1 + 2 + 3 by runs / so): tables of width 16, 4096 points 33 + 63 + 45 / 43 + 49 + 14, 4 x
// 50000 99 + 72 + 39 / 118 + 51 + 14; width 20 332 + 92 + 68 / 365 + 68 + 16.  With the doublings in one chain in
// k_weigh 43 + 25 + 45.  Pieces of 64 / 128 / 256 / 1024 buckets, lines + bits without doublings: at 4096 points 45 +
// 37 / 43 + 27 / 45 + 25 / 45 + 25, at width 20 547 + 338 / 434 + 176 / 375 + 96 / 357 + 53; k_bits with 32 / 64 quads
// there 53 / 43.
// In this form a window's seg_begin and nseg count its pieces of lines, grp_begin and ngrp its sums.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kLineQuads = 32, kBitQuads = 64;

// The sum of n points over the block's Q quads (valid in quad 0); point(i, live) sets live where there is
// one, else it returns the identity.  A warp with nothing to add skips the addition.
template <uint32_t Q, class F>
__device__ __forceinline__ fq_t block_line_sum(uint32_t n, uint4 *sh, F point) {
  __shared__ bool sh_live[Q];
  const uint32_t q = threadIdx.x >> 2;
  const uint32_t warp_q0 = (threadIdx.x >> 5) * 8;
  bool live = false, next_live = false;
  fq_t acc = point(q, live), next = point(q + Q, next_live);
#pragma unroll 1
  for (uint32_t i0 = Q; i0 < n; i0 += Q) {
    const fq_t b = next;
    const bool add = next_live;
    next_live = false;
    next = point(i0 + Q + q, next_live);
    if (__any_sync(kAllLanes, add)) acc = dq_add(acc, b, kAllLanes);
    live = live || add;
  }
  if (n <= 1) return acc;
  dq_store(sh + q * 12, acc);
  if ((threadIdx.x & 3) == 0) sh_live[q] = live;
  __syncthreads();
  uint32_t stride = Q / 2;
  while (stride >= n) stride >>= 1;  // quads from n on hold the identity
#pragma unroll 1
  for (; stride > 0; stride >>= 1) {
    fq_t o = dq_identity();
    bool add = false;
    if (q < stride) {
      o = dq_load(sh + (q + stride) * 12);
      add = sh_live[q + stride];
    }
    if (warp_q0 < stride && __any_sync(kAllLanes, add)) acc = dq_add(acc, o, kAllLanes);
    live = live || add;
    __syncthreads();
    if (q < stride) {
      dq_store(sh + q * 12, acc);
      if ((threadIdx.x & 3) == 0) sh_live[q] = live;
    }
    __syncthreads();
  }
  return acc;
}

__global__ void __launch_bounds__(4 * kLineQuads) k_lines(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  __shared__ uint4 sh[kLineQuads * 12];
  const WinDesc wd = pb.wins[find_win(pb.wins, pb.n_wins, blockIdx.x)];
  const Lines l = lines_of(wd.nb, pb.line_log2);
  uint32_t li = blockIdx.x - wd.seg_begin, b0, step, n;
  if (li < l.h * l.pr) {
    const uint32_t i0 = (li % l.pr) << pb.line_log2;
    b0 = ((li / l.pr) << l.wl) + i0;
    step = 1;
    n = min(l.w - i0, 1u << pb.line_log2);
  } else {
    li -= l.h * l.pr;
    const uint32_t i0 = (li % l.pc) << pb.line_log2;
    b0 = li / l.pc + (i0 << l.wl);
    step = l.w;
    n = min(l.h - i0, 1u << pb.line_log2);
  }
  const fq_t sum = block_line_sum<kLineQuads>(n, sh, [&](uint32_t i, bool &live) {
    const uint32_t b = b0 + i * step, gb = wd.bucket_begin + b;
    live = i < n && b < wd.nb && pb.count[gb] != 0;
    return live ? dq_load(pb.partials + (size_t)pb.taskoff[gb] * 12) : dq_identity();
  });
  if (threadIdx.x < 4) dq_store(pb.seg_out + (size_t)blockIdx.x * 12, sum);
}

__global__ void __launch_bounds__(4 * kBitQuads) k_bits(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  __shared__ uint4 sh[kBitQuads * 12];
  const WinDesc wd = pb.wins[find_win_grp(pb.wins, pb.n_wins, blockIdx.x)];
  const Lines l = lines_of(wd.nb, pb.line_log2);
  const uint32_t s = blockIdx.x - wd.grp_begin;
  const uint4 *rows = pb.seg_out + (size_t)wd.seg_begin * 12, *cols = rows + (size_t)l.h * l.pr * 12;
  const bool col = s < l.wl;
  const uint32_t bit = col ? s : s - l.wl, p = col ? l.pc : l.pr;
  const uint32_t n = (col ? l.w >> 1 : 1u << (l.hl - 1)) * p;
  const uint32_t more = s == l.wl ? l.pc : 0u;  // lo + 1 = W, the last column, counts as a row of bit 0
  const fq_t sum = block_line_sum<kBitQuads>(n + more, sh, [&](uint32_t i, bool &live) {
    if (i >= n + more) return dq_identity();
    live = true;
    if (i >= n) return dq_load(cols + ((size_t)(l.w - 1) * l.pc + (i - n)) * 12);
    const uint32_t e = i / p, j = ((e >> bit) << (bit + 1)) | (1u << bit) | (e & ((1u << bit) - 1u));
    if (col) return dq_load(cols + ((size_t)(j - 1) * p + i % p) * 12);
    return j < l.h ? dq_load(rows + ((size_t)j * p + i % p) * 12) : dq_identity();
  });
  if (threadIdx.x < 4) {  // 2^s times the sum: the blocks' doublings run side by side
    fq_t v = sum;
#pragma unroll 1
    for (uint32_t k = 0; k < s; k++) v = dq_dbl(v, 0xfu);
    dq_store(pb.grp_out + (size_t)blockIdx.x * 12, v);
  }
}

// One warp per window: the sum of its weighed sums.
__global__ void __launch_bounds__(32) k_weigh(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  const WinDesc wd = pb.wins[blockIdx.x];
  const uint32_t n = wd.ngrp, q = threadIdx.x >> 2;
  const uint4 *sums = pb.grp_out + (size_t)wd.grp_begin * 12;
  fq_t v = q < n ? dq_load(sums + (size_t)q * 12) : dq_identity();
#pragma unroll 1
  for (uint32_t k0 = 8; k0 < n; k0 += 8)
    v = dq_add(v, k0 + q < n ? dq_load(sums + (size_t)(k0 + q) * 12) : dq_identity(), kAllLanes);
#pragma unroll 1
  for (int d = 16; d >= 4; d >>= 1) {
    fq_t o;
#pragma unroll
    for (int j = 0; j < FQ_LIMBS; j++) o.v[j] = __shfl_down_sync(kAllLanes, v.v[j], d);
    // the quads past the end got their own point back: adding it would be a doubling
    v = dq_add(v, fq_select((int)threadIdx.x + d < 32, o, dq_identity()), kAllLanes);
  }
  if (threadIdx.x < 4) dq_store(pb.win_sum + (size_t)blockIdx.x * 12, v);
}

// ---------------------------------------------------------------------------------------------
// 6. buckets spread over several tasks: a quad per bucket of at most kMergeQuadMax runs (the common
//    case: a few more entries than seg_len), then a block of 64 quads per larger one (a value repeated
//    across many scalars): each quad sums a strided share of the partials, a tree over the quads in
//    shared memory the rest.  A thread, a warp or a block per bucket, in three kernels that each walked
//    the whole list, took (us, then now) 68 / 23 at 2^20 points, 386 / 72 in a shared pass of 4 x 50000
//    (121e3 split buckets), 364 / 103 in the uneven mix of 64.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kRedThreads) k_merge(PassBuffers pb) {
  pdl_begin();
  if (pb.counters[CNT_ERROR]) return;
  __shared__ uint4 sh[kRedQuads * 12];
  const uint32_t nsmall = pb.counters[CNT_HEAVY], nbig = pb.counters[CNT_BIG];
  const uint32_t mask = dq_mask();
  const uint32_t quads = gridDim.x * (blockDim.x / 4);
  for (uint32_t h = (blockIdx.x * blockDim.x + threadIdx.x) >> 2; h < nsmall; h += quads) {
    const uint32_t b = pb.heavy[h];
    const uint32_t nt = ntask_of(pb.count[b], pb);
    const uint32_t t0 = pb.taskoff[b];
    fq_t acc = dq_load(pb.partials + (size_t)t0 * 12);
#pragma unroll 1
    for (uint32_t k = 1; k < nt; k++) acc = dq_add(acc, dq_load(pb.partials + (size_t)(t0 + k) * 12), mask);
    dq_store(pb.partials + (size_t)t0 * 12, acc);
  }
  __syncthreads();
  const uint32_t q = threadIdx.x >> 2;
  const uint32_t warp_q0 = (threadIdx.x >> 5) * 8;  // first quad of this warp
  for (uint32_t h = blockIdx.x; h < nbig; h += gridDim.x) {
    const uint32_t b = pb.heavy[pb.n_buckets - 1 - h];
    const uint32_t nt = ntask_of(pb.count[b], pb);
    const uint32_t t0 = pb.taskoff[b];
    fq_t acc = q < nt ? dq_load(pb.partials + (size_t)(t0 + q) * 12) : dq_identity();
#pragma unroll 1
    for (uint32_t k0 = kRedQuads; k0 < nt; k0 += kRedQuads) {  // the same trip count for every quad
      const fq_t p = k0 + q < nt ? dq_load(pb.partials + (size_t)(t0 + k0 + q) * 12) : dq_identity();
      acc = dq_add(acc, p, kAllLanes);
    }
    dq_store(sh + q * 12, acc);
    __syncthreads();
#pragma unroll 1
    for (uint32_t stride = kRedQuads / 2; stride > 0; stride >>= 1) {
      fq_t o = dq_identity();
      if (q < stride) o = dq_load(sh + (q + stride) * 12);
      if (warp_q0 < stride) acc = dq_add(acc, o, kAllLanes);
      __syncthreads();
      if (q < stride) dq_store(sh + q * 12, acc);
      __syncthreads();
    }
    if (threadIdx.x < 4) dq_store(pb.partials + (size_t)t0 * 12, acc);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// 9. per MSM: window combine, Weierstrass map, special bases, ABI output
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void load_class_point(wpt_t &p, const uint4 *cp) {
  fq_load(p.x, cp);
  fq_load(p.y, cp + 3);
  p.z = fq_one();
}

__global__ void __launch_bounds__(128) k_final(PassBuffers pb) {
  pdl_begin();
  const uint32_t j = blockIdx.x;
  if (j >= pb.n_jobs) return;
  const JobDesc jd = pb.jobs[j];
  __shared__ uint32_t cls_sum[8];
  if (threadIdx.x < 8) cls_sum[threadIdx.x] = 0;
  __syncthreads();
  // multiples of the special bases: every special base has order 2 or 4 (y = 0, or
  // Montgomery u = -1), so k * P = (k mod 4) * P
  for (uint32_t s = threadIdx.x; s < pb.n_special; s += blockDim.x) {
    const uint32_t idx = pb.special_idx[s];
    if (idx < jd.base_off || idx >= jd.base_off + jd.n) continue;
    const uint4 w0 = pb.scalars[2 * (jd.scalar_off + (idx - jd.base_off))];
    atomicAdd(&cls_sum[pb.special_cls[s] & 7], w0.x & 3u);
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;  // warp 0 goes on: lanes 0..3 run the combine, all lanes the map
  uint64_t *out = pb.results + (size_t)jd.result_slot * 18;
  if (pb.counters[CNT_ERROR]) {
    if (threadIdx.x == 0)
      for (int k = 0; k < 18; k++) out[k] = 0;
    return;
  }
  // Horner over the windows: acc = 2^c * acc + WS_w (pippenger.h:36-45 doubles per offset)
  fq_t dacc = dq_identity();
  if (threadIdx.x < 4 && jd.n > 0 && jd.nred > 0) {
    dacc = dq_load(pb.win_sum + (size_t)(jd.win_begin + jd.nred - 1) * 12);
#pragma unroll 1
    for (int w = (int)jd.nred - 2; w >= 0; w--) {
#pragma unroll 1
      for (uint32_t k = 0; k < jd.c; k++) dacc = dq_dbl(dacc, 0xfu);
      dacc = dq_add(dacc, dq_load(pb.win_sum + (size_t)(jd.win_begin + w) * 12), 0xfu);
    }
  }
  __syncwarp();
  fq_t X, Y, Z;  // lane 0 holds X, 2 Y, 3 Z
#pragma unroll
  for (int k = 0; k < FQ_LIMBS; k++) {
    X.v[k] = __shfl_sync(kAllLanes, dacc.v[k], 0);
    Y.v[k] = __shfl_sync(kAllLanes, dacc.v[k], 2);
    Z.v[k] = __shfl_sync(kAllLanes, dacc.v[k], 3);
  }
  wpt_t res = te_to_weierstrass_warp(X, Y, Z);  // z is 1, or 0 for infinity
  if (threadIdx.x != 0) return;
  bool added = false;
  for (uint32_t c = 0; c < pb.n_classes && c < 8; c++) {
    const uint32_t m = cls_sum[c] & 3u;
    if (m == 0) continue;
    wpt_t p;
    load_class_point(p, pb.class_pts + c * 6);
    for (uint32_t k = 0; k < m; k++) res = w_add(res, p);
    added = true;
  }
  if (added) res = w_normalize(res);
  // g1_projective_t {x[6], y[6], z[6]}: (x*R, y*R, R) or arkworks' zero() (R, R, 0)
  const fq_t one = fq_canon(fq_one());
  const bool inf = fq_is_zero(res.z);
  const fq_t ox = inf ? one : fq_canon(res.x);
  const fq_t oy = inf ? one : fq_canon(res.y);
  const fq_t oz = inf ? fq_zero() : one;
  for (int k = 0; k < 6; k++) {
    out[k] = ((uint64_t)ox.v[2 * k + 1] << 32) | ox.v[2 * k];
    out[6 + k] = ((uint64_t)oy.v[2 * k + 1] << 32) | oy.v[2 * k];
    out[12 + k] = ((uint64_t)oz.v[2 * k + 1] << 32) | oz.v[2 * k];
  }
}

}  // namespace

// Scatter launches per pass: one per ~200 MB of sorted array, at most 8 (on GB300 the best
// counts measured were 4 for 2^24 points x 12 windows and 8 for 2^26 x 11 windows).
uint32_t msm_scatter_passes(uint64_t max_entries) {
  const uint64_t bytes = max_entries * 4, per = 200ull << 20;
  const uint64_t p = (bytes + per / 2) / per;
  return (uint32_t)(p < 1 ? 1 : p > 8 ? 8 : p);
}

// Key ranges of the ranked sort, as a shift of the bucket key (ranges of 2^shift keys, at most
// MSM_MAX_BINS of them).
//   * One MSM: one range per ~16 MB of sorted array, at most ten.  Measured on GB300 (scatter, us,
//     1 / 4 / 8 / 16 ranges): 2^20 points (13.6e6 entries) 146 / 125 / 135 / 162, 2^21 without tables
//     (31e6) 520 / 311 / 288 / 298, 3e6 (39e6) 490 / 383 / 350 / 353.
//   * Several MSMs (`many`): one range.  Each MSM's points and buckets are contiguous, so the blocks in
//     flight stay within one or two MSMs' slices by themselves.
// `ranges` > 0 asks for that many ranges instead (rounded to a shift).
uint32_t msm_bin_shift(uint32_t n_buckets, uint64_t max_entries, uint32_t ranges, bool many) {
  const uint64_t per = 16ull << 20;
  uint64_t want = ranges ? ranges : (max_entries * 4 + per / 2) / per;
  if (!ranges) want = many ? 1 : std::min<uint64_t>(want, 10);
  const uint32_t target = (uint32_t)(want < 1 ? 1 : want > MSM_MAX_BINS ? MSM_MAX_BINS : want);
  uint32_t shift = 0;
  while (shift < 31 && (((uint64_t)n_buckets + (1ull << shift) - 1) >> shift) > target) shift++;
  return shift;
}

// Points per chunk of a chunked scalar upload: a multiple of the histogram block, so every block
// of a chunk's histogram launch is a whole chunk of the stage.
uint64_t msm_upload_chunk_points(uint64_t n_points, int nchunks, uint32_t chunk_points) {
  const uint64_t per = (n_points + nchunks - 1) / nchunks;
  return (per + chunk_points - 1) / chunk_points * chunk_points;
}

size_t msm_partition_smem(uint32_t n_bins, uint32_t stage_cap) { return (size_t)n_bins * 4 + (size_t)stage_cap * 6; }

size_t msm_scan_tmp_words(uint32_t n_buckets) {
  return 2ull * ((n_buckets + kScanBlock - 1) / kScanBlock) + 2;
}

// Level-1 reductions of at most this many runs take a quad each (k_reduce1_quad): one thread each
// would leave the GPU idle behind a chain of 8 products per addition.  Measured on GB300 (us per call, threads /
// quads): 4 MSMs of 4096 points on plain records (12 K runs) 929 / 879, 65536 points there (10 K) 1238 / 1176, 17 MSMs of
// 50000 points on width 16 (35 K) 3670 / 3692.  Far above the line the two are within a few percent: 2^24 points (76 K
// runs of 64 buckets) 46.11 / 45.80 ms, 64 MSMs of 1000 points (131 K of 16) 1954 / 1863.
constexpr uint32_t kReduceQuadSegs = 32768;

cudaError_t msm_launch_pass(const PassBuffers &pb, int num_sms, cudaStream_t st, cudaEvent_t *ev,
                            const cudaEvent_t *chunk_ready, int nchunks, uint32_t *n_kernels) {
  cudaError_t e;
  uint32_t launched = 0;
  auto mark = [&](int k) {
    if (ev) cudaEventRecord(ev[k], st);
  };
  // one launch: kernel k on `grid` blocks, dependent on the one before it (see pdl_wait)
  cudaError_t bad = cudaSuccess;
  bool dependent = true;
  auto run = [&](auto k, uint32_t grid, uint32_t block, size_t smem, auto... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    const cudaError_t r = cudaLaunchKernelEx(&cfg, k, args...);
    if (r != cudaSuccess && bad == cudaSuccess) bad = r;
    launched++;
  };
  run(k_clear, std::min<uint32_t>(num_sms * 8, pb.n_buckets / 1024 + 1), 256, 0, pb);
  mark(0);
  const uint32_t pts_blocks = (uint32_t)((pb.n_points + 255) / 256);
  const size_t part_smem = msm_partition_smem(pb.n_bins, pb.stage_cap);
  const size_t place_smem = ((1u << pb.bin_shift) + 2 * kPlaceChunks + 1) * 4;
  if (pb.n_points > 0 && pb.bin_total) {
    // the limits are the kernels', not the pass's: another thread may be launching them too
    const auto limit = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = cudaFuncSetAttribute(k_partition, limit, MSM_PARTITION_SMEM)) ||
        (e = cudaFuncSetAttribute(k_place_count, limit, (int)kPlaceSmemMax)) ||
        (e = cudaFuncSetAttribute(k_place, limit, (int)kPlaceSmemMax)))
      return e;
    const uint64_t per = chunk_ready && nchunks > 0
                             ? msm_upload_chunk_points(pb.n_points, nchunks, pb.chunk_points) : pb.n_points;
    for (uint64_t g0 = 0, c = 0; g0 < pb.n_points; g0 += per, c++) {
      const uint64_t g1 = std::min(g0 + per, pb.n_points);
      if (chunk_ready && (e = cudaStreamWaitEvent(st, chunk_ready[c], 0))) return e;
      run(k_partition, (uint32_t)((g1 - g0 + pb.chunk_points - 1) / pb.chunk_points), kPartThreads, part_smem, pb,
          g0, g1);
    }
    run(k_place_count, pb.place_blocks, kPlaceThreads, place_smem, pb);
  } else if (pb.n_points > 0) {
    if (chunk_ready && nchunks > 0) {
      // the scalars arrive in chunks on another stream: count each chunk as soon as it lands
      const uint64_t per = msm_upload_chunk_points(pb.n_points, nchunks, MSM_POINTS_PER_CHUNK);
      for (int c = 0; c < nchunks; c++) {
        const uint64_t g0 = (uint64_t)c * per, g1 = g0 + per < pb.n_points ? g0 + per : pb.n_points;
        if ((e = cudaStreamWaitEvent(st, chunk_ready[c], 0))) return e;
        if (g1 > g0) run(k_count, (uint32_t)((g1 - g0 + 255) / 256), 256, 0, pb, g0, g1);
      }
    } else {
      run(k_count, pts_blocks, 256, 0, pb, 0, pb.n_points);
    }
  }
  mark(1);
  const uint32_t nblk = (pb.n_buckets + kScanBlock - 1) / kScanBlock;
  const bool scan_small = nblk <= kScanSmallBlocks;
  if (nblk > 0 && scan_small) {
    run(k_scan_small, nblk, kScanThreads, (pb.seg_len + 1) * 4, pb);
  } else if (nblk > 0) {
    run(k_scan_reduce, nblk, kScanThreads, 0, pb);
    run(k_scan_blocks, 1, kScanThreads, 0, pb, nblk);
    run(k_scan_apply, nblk, kScanThreads, 0, pb);
  }
  mark(2);
  if (pb.n_points > 0 && pb.bin_total) {
    run(k_place, pb.place_blocks, kPlaceThreads, place_smem, pb);
  } else if (pb.n_points > 0 && pb.stage) {
    // few chunks: several blocks each (a block walks a chunk of 256 points in ~17 dependent steps; 4096
    // points, 16 chunks: 12.8 us with a block each, 4.6 with eight)
    const uint32_t parts = std::max(1u, std::min(8u, (uint32_t)num_sms * 16u / pts_blocks));
    for (uint32_t r = 0; r < pb.n_bins; r++) run(k_scatter_staged, pts_blocks * parts, 256, 0, pb, r, parts);
  } else if (pb.n_points > 0) {
    const uint32_t passes = msm_scatter_passes(pb.max_entries);
    for (uint32_t p = 0; p < passes; p++) {
      const uint32_t lo = (uint32_t)((uint64_t)pb.n_buckets * p / passes);
      const uint32_t hi = (uint32_t)((uint64_t)pb.n_buckets * (p + 1) / passes);
      run(k_scatter, pts_blocks, 256, 0, pb, lo, hi);
    }
  }
  mark(3);
  if (pb.n_buckets > 0) {
    if (!scan_small) run(k_len_hist, num_sms * 4, 256, (pb.seg_len + 1) * 4, pb);
    run(k_tasks, (pb.n_buckets + 255) / 256, 256, 2 * (pb.seg_len + 1) * 4, pb);
  }
  mark(4);
  // Fewer blocks than an SM holds (a server's passes) start when k_tasks has left: set up beside its
  // blocks they would share some SMs four by four and leave others with two.  Measured on GB300, three
  // per SM: 2^20 points 4.50 ms set up early, 3.72 ms so.
  dependent = !pb.acc_blocks_per_sm;
  const uint32_t acc_blocks = num_sms * (pb.acc_blocks_per_sm ? pb.acc_blocks_per_sm : 4);
  if (pb.quads)
    run(k_accumulate_quad, acc_blocks, 128, 0, pb);
  else
    run(k_accumulate, acc_blocks, 128, 0, pb);
  dependent = true;
  mark(5);
  run(k_merge, num_sms * 2, kRedThreads, 0, pb);
  mark(6);
  if (pb.lines && pb.n_segs > 0) {
    run(k_lines, pb.n_segs, 4 * kLineQuads, 0, pb);
  } else if (pb.n_segs > 0) {
    if (pb.n_segs <= kReduceQuadSegs)
      run(k_reduce1_quad, (pb.n_segs + 31) / 32, 128, 0, pb);
    else
      run(k_reduce1, (pb.n_segs + 127) / 128, 128, 0, pb);
  }
  mark(7);
  // Level 2 in blocks of 256 threads; level 3 (one block per window of more than 16 groups) in blocks of 128
  // while they fit on the SMs in one wave: with one warp per SMSP a quad addition takes 1.9 us, with two 2.8,
  // but a quad of the smaller block sums twice as many runs in sequence.  Measured on GB300 (us, 256 / 128
  // threads): level 2 of 4 MSMs of 4096 points on plain records 66 / 68, of 32 of 1000 on width 16 133 / 158, of
  // 64 of those 256 / 201, of 2^24 points 135 / 160; level 3 of 2^24 points (150 groups) 88 / 100.
  if (pb.lines && pb.n_grps > 0) {
    run(k_bits, pb.n_grps, 4 * kBitQuads, 0, pb);
  } else if (pb.n_grps > 0) {
    run(k_reduce2, pb.n_grps, kRedThreads, 0, pb);
  }
  mark(8);
  if (pb.lines && pb.n_wins > 0) {
    run(k_weigh, pb.n_wins, 32, 0, pb);
  } else if (pb.n_wins > 0) {
    if (pb.min_grps <= kRed3SmallMax) run(k_reduce3_small, (pb.n_wins + 31) / 32, 128, 0, pb);
    if (pb.max_grps <= kRed3SmallMax) {
      // no window for k_reduce3
    } else if (pb.n_wins <= (uint32_t)num_sms)
      run(k_reduce3<128>, pb.n_wins, 128, 0, pb);
    else
      run(k_reduce3<256>, pb.n_wins, 256, 0, pb);
  }
  mark(9);
  if (pb.n_jobs > 0) {
    run(k_final, pb.n_jobs, 128, 0, pb);
  }
  mark(10);
  if (n_kernels) *n_kernels = launched;
  return bad != cudaSuccess ? bad : cudaGetLastError();
}

// The cluster row sampler: one row per thread-block CLUSTER, any element type, alignment, vocabulary and knobs, every output.
//
// A row is cut into as many contiguous slices as its cluster has blocks (16 for a handful of rows, 1 for a batch that fills the
// GPU by itself), so one row is spread over 16 SMs and a batch of 64 over 256 blocks, two to an SM; the blocks exchange through distributed shared
// memory and the hardware cluster barrier (well under a microsecond), in ONE launch. Per row:
//
//   load       every block reads its slice once (kept in shared memory as binary32 when it fits, else read again from L2): maximum,
//              its lowest index, smallest finite logit, maxima of groups; odd values (NaN, +inf, BF16 below 2^-39) send the row to the generic code
//   histogram  1024 bins, linear in the logit below the row's maximum: counts (a top_k wants them), fixed-point sums of
//              exp((z - vmax) / T) in FP64 (a top-p over binary32 values wants them), or of the draw's integer weights. The bins of
//              the blocks are added up, a share by every block, and pushed to all of them
//   crossing   every block walks the bins (block scan) to the bin where a count or mass is reached; the logits of that one bin (a few
//              hundred), or with a top_k every logit down to that bin, are gathered into a list in every block's shared memory and
//              put in order; the exact threshold is found on them
//   draw       the same walk on the integer weights, down to the bin, then inside its ordered list; or the Gumbel keys of the kept
//              logits, where a logit is given the two logarithms only if its noise can beat the best key known so far
//
// Every block of the cluster comes to the same decisions from the same numbers, so no block waits for another's verdict and rank
// 0 writes the outputs. What cannot be decided here (a list that overflows, a mass closer to its target than its error bound) goes to
// sample_row_generic, run by rank 0.
//
// Exactness: integer weights, counts and list order are exact. The top-p target is p * total with total and the mass above the
// crossing bin either fixed-point FP64 exponentials (rounded to 2^-44, so off by at most n 2^-44 for n logits) or, for BF16
// values, sums of the integer weights (whose bound kWeightBand derives), or, with a top_k, an FP32 sum (the bound of sample_topk.cuh):
// a boundary inside that bound is decided again with the next finer sums. Inside the list the masses are FP64.
//
// What bounds it: the latency of ~6 barrier-separated phases for a few rows; for a batch the FP64 pipe (14 operations per logit) on
// rows without a top_k and the shared-memory atomics on the others.
// No counterpart in the reference (kernels/common/sample.metal:34-198 spreads a row over threadgroups with device-memory histograms).
#pragma once
#include <cfloat>
#include <cstddef>

#include "common.cuh"
#include "sample_generic.cuh"
#include "sample_topk.cuh"
#include "vocab_parallel.cuh"

namespace lm {

constexpr int kCBins = 1024;
constexpr int kCList = 2048;             // logits of one gathered list
constexpr int kCListK = 1024;            // largest top_k whose whole set is gathered
constexpr int kCGroups = 4096;           // group maxima per block
constexpr int kCMaxBins = 512;           // bins of the group maxima
constexpr int kCMaxRanks = 16;           // blocks of one cluster
constexpr int kCQueue = 128;             // logits a warp's queue of the Gumbel draw holds
constexpr uint32_t kCallOrdered = 1u, kCallFew = 2u;   // of a launch: the rows are taken by kind; a call of a few rows with one top_k (LM_STATUS_SLICED_PATH)
constexpr int kOrderRows = 2048;         // rows whose order a block looks up (row_in_order)
// A list up to this long is ordered by counting larger keys, a longer one by bins first (472 keys: 7.7 us by counting, 1.5 by bins). us a call of 12 FP32 rows, by counting / by bins:
// top_k 64 15.16 / 15.44, 80 16.10 / 16.33, 100 16.38 / 16.46, 120 16.63 / 16.50, 140 16.98 / 16.58. A list of few distinct values (BF16 logits of one crossing bin, penalised or not) fills few bins, and
// the order inside those is counted all the same: by bins from where counting has a thread per key (inverse CDF, no top_k, means of 16 inputs, by counting to 320 / to 110 / to 256: 4 rows
// of 248,320 42.4 / 44.1 / 42.5, 45 of 53,442 53.6 / 54.7 / 53.8, one of 151,936 28.8 / 31.0 / 28.5 and, with longer lists, 32.5 / 31.5 / 31.0; penalised 29.4 / 31.9 / 29.2).
constexpr int kCRankOrder = 110, kCRankOrderFew = 256;
constexpr double kCMassBand = 1e-11;     // relative error of a logit's fixed-point softmass beyond its rounding: 7e-12 of the polynomial, a few 1e-16
// Threads per block: a block-wide reduction costs shuffles in proportion to its warps (1024 threads: 0.5 us each, measured), so no more
// warps than the sweeps need.
constexpr int kClusterBlock = 512;

// ---- the row as the kernel sees it -----------------------------------------------------------------------------------------------
// Chunks of eight elements counted from an address that 16-byte loads can take: element i of the row is element (i + off) % 8 of chunk
// (i + off) / 8. The first and the last chunk may be partial; positions outside the row read as -inf, which no phase counts.
struct ClusterRow {
  const char* row; int V, off, c0, c1;        // this block's chunks [c0, c1)
  const float4* vals; int nv;                  // cached: the slice's logits (penalised), elements 0-3 of chunk c at [c - c0], 4-7 at [nv + c - c0]
  const uint8_t* pen; float rho, pi;           // a byte per chunk: which of its elements are penalised (nullptr: none)
};


struct ClusterSmem {
  union {
    struct { uint32_t cnt[kCBins], lo[2][kCBins], hi[2][kCBins]; };        // this block's slice: counts; two 64-bit sums as two words each
    struct { unsigned long long list[kCList], sorted[kCList]; uint32_t fill[kCList]; };   // after the bins have been added up
    struct { double cum[kCList]; unsigned long long sorted_[kCList]; };    // (the gathered list is dead once it is in order)
    struct { unsigned long long list_[kCList]; uint32_t x_max[kCMaxRanks][kCMaxBins / 2]; uint32_t max_cnt[kCMaxBins]; };   // top_k: counts of the group maxima, 16 bits each
    struct { float2 queue[32][kCQueue]; };                                  // Gumbel draw: a warp's logits that wait for a hash
  };
  uint32_t r_cnt[kCBins + 4];            // the row's counts, then their exclusive running sum
  union {
    unsigned long long r_sum[2][kCBins]; // the row's sums (0: softmass, 1: draw weights), then their inclusive running sums
    double bin_exp[kCBins];              // while the bins are filled: the exp of a bin's centre
    float gmax[kCGroups];                // while the row is read: maxima of groups of its logits
  };
  double exp_tab[64];                    // 2^(i/64)
  // what the blocks of the cluster leave in one another's copy
  unsigned long long x_best[kCMaxRanks]; float x_low[kCMaxRanks], x_glow[kCMaxRanks]; uint32_t x_flags[kCMaxRanks];
  double x_mass[kCMaxRanks], x_mass64[kCMaxRanks], x_kept[kCMaxRanks];
  unsigned long long x_key[kCMaxRanks]; float x_rival[kCMaxRanks];
  uint32_t list_n[2];
  uint64_t scratch[32];
  double warp_d[32]; float warp_f[32], warp_g[32];
  uint32_t hit, hit2, pick; int token, amb;
  // The row, its knobs and what is known about it: the same for every thread, and kept here so that no thread holds them in registers
  // from phase to phase (a spill is a trip to L2: the kernel's shared memory leaves next to no L1).
  ClusterRow R;
  uint64_t seed; uint32_t step;
  double inv_t; float T, top_p, min_p, c2, vmax, vmin, gmin, scale; int top_k, arg, row, rank, C, window, every, per;
  uint32_t draw, flags; bool few, has_k, has_p, has_m, in_topk, inverse, want_w, want_stats, fallback;
  uint32_t t_id; float u;
  // results
  float o_tau; int o_token; uint32_t o_status; uint64_t o_weight; double kept_mass;
  alignas(16) uint32_t totals[kCMaxBins];
};
static_assert(offsetof(ClusterSmem, totals) % 16 == 0 && offsetof(ClusterSmem, bin_exp) % 16 == 0 && offsetof(ClusterSmem, queue) % 8 == 0, "16-byte accesses");

// ---- the cluster -------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  return r;
}
__device__ __forceinline__ void cst_u32(uint32_t a, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void cst_u64(uint32_t a, unsigned long long v) { asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ uint32_t cld_u32(uint32_t a) { uint32_t v; asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory"); return v; }
__device__ __forceinline__ uint32_t catom_add(uint32_t a, uint32_t v) { uint32_t o; asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory"); return o; }
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// All threads of all blocks of the cluster; writes before it are seen after it.
__device__ __forceinline__ void cluster_sync(int C) {
  if (C == 1) { __syncthreads(); return; }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 2^43 * e rounded to the nearest integer, 0 <= e <= 1: adding 2^9 leaves an ulp of 2^-43 in the sum's low bits.
__device__ __forceinline__ unsigned long long fixed43(double e) {
  return static_cast<unsigned long long>(__double_as_longlong(__dadd_rn(e, 512.0)) - 0x4080000000000000ll);
}

template <bool F32> struct RawChunk { uint4 a[F32 ? 2 : 1]; };

template <bool F32>
__device__ __forceinline__ RawChunk<F32> load_raw(const ClusterRow& R, int c) {
  RawChunk<F32> q;
  const int base = 8 * c - R.off;
  if (base >= 0 && base + 8 <= R.V) {
    const uint4* p = reinterpret_cast<const uint4*>(R.row + static_cast<int64_t>(base) * (F32 ? 4 : 2));
#pragma unroll
    for (int j = 0; j < (F32 ? 2 : 1); j++) q.a[j] = __ldg(p + j);
  } else {
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int i = base + e;
      const bool in = i >= 0 && i < R.V;
      w[e] = F32 ? (in ? __ldg(reinterpret_cast<const uint32_t*>(R.row) + i) : 0xFF800000u)
                 : (in ? static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(R.row) + i)) : 0xFF80u);
    }
    if (F32) { q.a[0] = make_uint4(w[0], w[1], w[2], w[3]); q.a[F32 ? 1 : 0] = make_uint4(w[4], w[5], w[6], w[7]); }
    else q.a[0] = make_uint4(w[0] | (w[1] << 16), w[2] | (w[3] << 16), w[4] | (w[5] << 16), w[6] | (w[7] << 16));
  }
  return q;
}
template <bool F32>
__device__ __forceinline__ void widen_raw(const ClusterRow& R, const RawChunk<F32>& q, int c, float z[8]) {
  if (F32) {
    z[0] = __uint_as_float(q.a[0].x); z[1] = __uint_as_float(q.a[0].y); z[2] = __uint_as_float(q.a[0].z); z[3] = __uint_as_float(q.a[0].w);
    const uint4 b = q.a[F32 ? 1 : 0];
    z[4] = __uint_as_float(b.x); z[5] = __uint_as_float(b.y); z[6] = __uint_as_float(b.z); z[7] = __uint_as_float(b.w);
  } else {
    const uint4 a = q.a[0];
    z[0] = bf16_lo(a.x); z[1] = bf16_hi(a.x); z[2] = bf16_lo(a.y); z[3] = bf16_hi(a.y);
    z[4] = bf16_lo(a.z); z[5] = bf16_hi(a.z); z[6] = bf16_lo(a.w); z[7] = bf16_hi(a.w);
  }
  if (R.pen) {
    const uint32_t bits = R.pen[c - R.c0];
    if (bits) {
#pragma unroll
      for (int e = 0; e < 8; e++) if ((bits >> e) & 1u) z[e] = penalise(z[e], R.rho, R.pi);
    }
  }
}
// f(c, z) for every chunk of this block's slice. Uncached, a few chunks per thread are in flight while f works on one.
template <bool F32, bool CACHED, class F>
__device__ __forceinline__ void sweep(const ClusterRow& R, F f) {
  const int B = static_cast<int>(blockDim.x);
  int c = R.c0 + static_cast<int>(threadIdx.x);
  if (CACHED) {
#pragma unroll 1
    for (; c < R.c1; c += B) {
      const float4 a = R.vals[c - R.c0], b = R.vals[R.nv + c - R.c0];
      const float z[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      f(c, z);
    }
  } else {
    constexpr int kDeep = F32 ? 2 : 4;
    RawChunk<F32> q[kDeep];
#pragma unroll
    for (int j = 0; j < kDeep; j++) if (c + j * B < R.c1) q[j] = load_raw<F32>(R, c + j * B);
#pragma unroll 1
    for (; c < R.c1; c += B) {
      const RawChunk<F32> now = q[0];
#pragma unroll
      for (int j = 0; j + 1 < kDeep; j++) q[j] = q[j + 1];
      if (c + kDeep * B < R.c1) q[kDeep - 1] = load_raw<F32>(R, c + kDeep * B);
      float z[8];
      widen_raw<F32>(R, now, c, z);
      f(c, z);
    }
  }
}

// The bin of a logit: 0 at the maximum, growing downwards; non-increasing in z because every step of it is monotone (explicitly
// rounded operations: every call site gives the same bin). The integer is read out of the sum with 2^23. With a window, only the
// logits of one such bin are looked at, and the bins divide it once more (kCBins: a logit outside the window).
constexpr int kLogBins = -2;             // ClusterBins::window: bins by the depth's exponent and four bits (2^-32 .. 2^32; what lies beyond shares the end bins)
constexpr uint32_t kLogBase = (127u - 32u) << 4;
__device__ __forceinline__ float log_bin_edge(uint32_t b) { return b == 0u ? 0.0f : b >= static_cast<uint32_t>(kCBins) ? INFINITY : __uint_as_float((b + kLogBase) << 19); }
struct ClusterBins {
  float vmax, scale; int window;                                            // -1: none; kLogBins; 0 .. kCBins - 1: a linear bin; kCBins + b: bin b of those by exponent
  __device__ __forceinline__ float depth(float z) const { return fminf(__fmul_rn(__fsub_rn(vmax, z), scale), static_cast<float>(kCBins - 1)); }
  __device__ __forceinline__ uint32_t coarse(float z) const { return __float_as_uint(__fadd_rn(depth(z), 8388608.0f)) & static_cast<uint32_t>(kCBins - 1); }
  __device__ __forceinline__ uint32_t by_exponent(float z) const {
    return min(max(__float_as_uint(__fsub_rn(vmax, z)) >> 19, kLogBase) - kLogBase, static_cast<uint32_t>(kCBins - 1));
  }
  __device__ __forceinline__ uint32_t of(float z) const {
    if (window == -1) return coarse(z);
    if (window == kLogBins) return by_exponent(z);
    if (window >= kCBins) {
      const uint32_t lb = static_cast<uint32_t>(window - kCBins);
      if (by_exponent(z) != lb) return kCBins;
      const float lo = log_bin_edge(lb), width = log_bin_edge(lb + 1u) - lo;   // (an infinite width, or a NaN product of it: bin 0)
      const float t = __fmul_rn(__fsub_rn(__fsub_rn(vmax, z), lo), __fdiv_rn(static_cast<float>(kCBins - 1), width));
      return __float_as_uint(__fadd_rn(fminf(fmaxf(t, 0.0f), static_cast<float>(kCBins - 1)), 8388608.0f)) & static_cast<uint32_t>(kCBins - 1);
    }
    if (coarse(z) != static_cast<uint32_t>(window)) return kCBins;
    const float t = __fmul_rn(__fsub_rn(depth(z), static_cast<float>(window) - 0.5f), static_cast<float>(kCBins - 1));
    return __float_as_uint(__fadd_rn(fminf(fmaxf(t, 0.0f), static_cast<float>(kCBins - 1)), 8388608.0f)) & static_cast<uint32_t>(kCBins - 1);
  }
};
__device__ __forceinline__ void bin_add_u64(uint32_t* lo, uint32_t* hi, uint32_t b, unsigned long long w) {
  const uint32_t wl = static_cast<uint32_t>(w);
  uint32_t wh = static_cast<uint32_t>(w >> 32);
  if (wl) { const uint32_t old = atomicAdd(&lo[b], wl); wh += (old + wl < old) ? 1u : 0u; }
  if (wh) atomicAdd(&hi[b], wh);
}
// Four at once: the low words' replies (the carries) are all awaited together, one trip to the shared memory's atomic unit instead of four.
__device__ __forceinline__ void bin_add4_u64(uint32_t* lo, uint32_t* hi, const uint32_t (&b)[4], const uint64_t (&w)[4]) {
  uint32_t old[4];
#pragma unroll
  for (int e = 0; e < 4; e++) { const uint32_t wl = static_cast<uint32_t>(w[e]); old[e] = 0u; if (wl) old[e] = atomicAdd(&lo[b[e]], wl); }
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const uint32_t wl = static_cast<uint32_t>(w[e]), wh = static_cast<uint32_t>(w[e] >> 32) + (old[e] + wl < old[e] ? 1u : 0u);
    if (wh) atomicAdd(&hi[b[e]], wh);
  }
}

// ---- block-wide reductions whose second stage is one warp's (a shuffle costs every warp that issues it: one per cycle and SM) ---------
__device__ __forceinline__ double cblock_sum_f64(double v, uint64_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* d = reinterpret_cast<double*>(scratch);
  v = warp_sum_f64(v);
  if (lane == 0) d[warp] = v;
  __syncthreads();
  if (warp == 0) { const double r = warp_sum_f64(lane < nw ? d[lane] : 0.0); __syncwarp(); if (lane == 0) d[31] = r; }
  __syncthreads();
  return d[31];
}
__device__ __forceinline__ uint64_t cblock_sum_u64(uint64_t v, uint64_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum_u64(v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) { const uint64_t r = warp_sum_u64(lane < nw ? scratch[lane] : 0ull); __syncwarp(); if (lane == 0) scratch[31] = r; }
  __syncthreads();
  return scratch[31];
}
__device__ __forceinline__ uint64_t cblock_max_u64(uint64_t v, uint64_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_max_u64(v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) { const uint64_t r = warp_max_u64(lane < nw ? scratch[lane] : 0ull); __syncwarp(); if (lane == 0) scratch[31] = r; }
  __syncthreads();
  return scratch[31];
}
// Exclusive running sum over the threads; *total gets the sum. (At most 31 warps: scratch[31] is the total.)
__device__ __forceinline__ uint64_t cblock_scan_u64(uint64_t v, uint64_t* scratch, uint64_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint64_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint64_t w = lane < nw ? scratch[lane] : 0ull;
    uint64_t x = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, x, o); if (lane >= o) x += t; }
    __syncwarp();
    if (lane < nw) scratch[lane] = x - w;
    if (lane == 31) scratch[31] = x;
  }
  __syncthreads();
  if (total) *total = scratch[31];
  return scratch[warp] + incl - v;
}
__device__ __forceinline__ uint32_t cblock_scan_u32(uint32_t v, uint64_t* scratch64, uint32_t* total) {
  uint32_t* scratch = reinterpret_cast<uint32_t*>(scratch64);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < nw ? scratch[lane] : 0u;
    uint32_t x = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(kFull, x, o); if (lane >= o) x += t; }
    __syncwarp();
    if (lane < nw) scratch[lane] = x - w;
    if (lane == 31) scratch[31] = x;
  }
  __syncthreads();
  if (total) *total = scratch[31];
  return scratch[warp] + incl - v;
}

// ---- block-wide steps on the bins and lists ----------------------------------------------------------------------------------------
// Inclusive running sum over the bins, in place.
template <int B>
static __device__ __noinline__ void scan_bins(unsigned long long* a, uint64_t* scratch) {
  constexpr int kPer = kCBins / B;
  uint64_t v[kPer], s = 0ull;
#pragma unroll
  for (int j = 0; j < kPer; j++) { s += a[threadIdx.x * kPer + j]; v[j] = s; }
  const uint64_t before = cblock_scan_u64(s, scratch, nullptr);
#pragma unroll
  for (int j = 0; j < kPer; j++) a[threadIdx.x * kPer + j] = before + v[j];
  __syncthreads();
}
// The counts' exclusive running sum in place, the total behind the last bin.
template <int B>
static __device__ __noinline__ void scan_counts(uint32_t* a, uint64_t* scratch) {
  constexpr int kPer = kCBins / B;
  uint32_t v[kPer], sum = 0u;
#pragma unroll
  for (int j = 0; j < kPer; j++) { v[j] = sum; sum += a[threadIdx.x * kPer + j]; }
  uint32_t total = 0u;
  const uint32_t before = cblock_scan_u32(sum, scratch, &total);
#pragma unroll
  for (int j = 0; j < kPer; j++) a[threadIdx.x * kPer + j] = before + v[j];
  if (threadIdx.x == 0) a[kCBins] = total;
  __syncthreads();
}
// Inclusive FP64 running sum over v[0 .. n) in place, index order (the warps' totals are scanned by every warp for itself).
template <int B>
static __device__ __noinline__ void scan_list_f64(double* v, int n, double* warp_d) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double carry = 0.0;
  for (int base = 0; base < n; base += B) {
    const int i = base + static_cast<int>(threadIdx.x);
    double x = 0.0;
    if (base + warp * 32 < n) {                                             // only the warps that hold something
      x = i < n ? v[i] : 0.0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const double t = __shfl_up_sync(kFull, x, o); if (lane >= o) x += t; }
    }
    if (lane == 31) warp_d[warp] = x;
    __syncthreads();
    if (warp == 0) {
      const double w = lane < B / 32 ? warp_d[lane] : 0.0;
      double t = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const double q = __shfl_up_sync(kFull, t, o); if (lane >= o) t += q; }
      __syncwarp();
      const double before = __shfl_up_sync(kFull, t, 1);
      if (lane < B / 32) warp_d[lane] = lane ? before : 0.0;
      if (lane == 31) warp_d[31] = t;
    }
    __syncthreads();
    if (i < n) v[i] = carry + warp_d[warp] + x;
    carry += warp_d[31];
    __syncthreads();
  }
}
// Orders list[0 .. n) (distinct keys, values between bottom and top) descending into sorted[]; every thread calls. in_bins: the values of a bin of the list's span are
// equal and their indices may come in any order, so that the bins alone do (4 rows of 248,320 BF16 logits, a list of 370: 5.9 us by rank inside the bins one key at a time, 4.2 eight at a time, 1.2 so).
template <int B>
static __device__ __noinline__ void order_list(ClusterSmem& s, int n, float top, float bottom, bool in_bins = false, int by_rank = kCRankOrder) {
  const int tid = threadIdx.x;
  if (n <= by_rank) {                                                       // by counting the larger keys, several threads to a key
    for (int i = tid; i < n; i += B) s.fill[i] = 0u;
    __syncthreads();
    const int parts = n > 0 ? B / n : 1, e = tid / parts, p = tid - e * parts;
    if (e < n) {
      const unsigned long long k = s.list[e];
      uint32_t r = 0u;
#pragma unroll 4
      for (int j = p; j < n; j += parts) r += s.list[j] > k ? 1u : 0u;
      if (r) atomicAdd(&s.fill[e], r);
    }
    __syncthreads();
    for (int i = tid; i < n; i += B) s.sorted[s.fill[i]] = s.list[i];
    __syncthreads();
    return;
  }
  // a counting sort over bins of the list's own span, then by rank inside a bin
  const ClusterBins lb{top, static_cast<float>(kCBins - 1) / (top > bottom ? top - bottom : 1.0f), -1};
  uint32_t* off = s.fill;                                                   // [kCBins] running sums ...
  uint32_t* put = s.fill + kCBins;                                          // ... [kCBins] how many have been put
  for (int i = tid; i < 2 * kCBins; i += B) s.fill[i] = 0u;
  __syncthreads();
  for (int i = tid; i < n; i += B) atomicAdd(&off[lb.coarse(fkey_inv(static_cast<uint32_t>(s.list[i] >> 32)))], 1u);
  __syncthreads();
  {
    constexpr int kPer = kCBins / B;
    uint32_t v[kPer], sum = 0u;
#pragma unroll
    for (int j = 0; j < kPer; j++) { v[j] = sum; sum += off[tid * kPer + j]; }
    const uint32_t before = cblock_scan_u32(sum, s.scratch, nullptr);
#pragma unroll
    for (int j = 0; j < kPer; j++) off[tid * kPer + j] = before + v[j];
  }
  __syncthreads();
  for (int i = tid; i < n; i += B) {
    const unsigned long long key = s.list[i];
    const uint32_t b = lb.coarse(fkey_inv(static_cast<uint32_t>(key >> 32)));
    s.sorted[off[b] + atomicAdd(&put[b], 1u)] = key;
  }
  __syncthreads();
  if (in_bins) return;
  for (int i = tid; i < n; i += B) {
    const unsigned long long key = s.sorted[i];
    const uint32_t b = lb.coarse(fkey_inv(static_cast<uint32_t>(key >> 32)));
    const uint32_t lo = off[b], hi = lo + put[b];
    uint32_t r = lo;
#pragma unroll 8
    for (uint32_t j = lo; j < hi; j++) r += s.sorted[j] > key ? 1u : 0u;
    s.list[r] = key;
  }
  __syncthreads();
  for (int i = tid; i < n; i += B) s.sorted[i] = s.list[i];
  __syncthreads();
}

// How far the sums of integer weights (times 2^-40) can be from the exact masses, relative to the row's mass Z >= 1 (n logits, u = 2^-24):
// the rounded (z - vmax), their product with c and c itself each move an exponent x by at most u |x|, and the terms' weighted |x ln2| is at most
// ln n (sample_topk.cuh gives the argument): 3 u ln n; spec_exp2 is within 1.7e-7; dropping the fraction costs at most 2^-40 a term.
__device__ __forceinline__ double weight_band(int n) { return 1.25 * (3.0 * 5.9604644775390625e-8 * log(static_cast<double>(n)) + 1.7e-7); }

// ---- the phases, each a function of its own: its loop gets the registers, and its code exists once ------------------------------------
static __device__ __noinline__ void generic_row_fallback(const SampleDev& P0, const ClusterSmem& s, unsigned char* smem) {
  SampleDev P = P0;
  P.seed = s.seed; P.step = s.step;
  const int row = s.row;
  __syncthreads();                                                          // (s is written over)
  sample_row_generic(P, row, *reinterpret_cast<GenericSmem*>(smem), reinterpret_cast<uint32_t*>(smem + sizeof(GenericSmem)));
}

__device__ __forceinline__ float pick8(const float (&z)[8], int e) {
  const float a = (e & 1) ? z[1] : z[0], b = (e & 1) ? z[3] : z[2], c = (e & 1) ? z[5] : z[4], d = (e & 1) ? z[7] : z[6];
  const float l = (e & 2) ? b : a, h = (e & 2) ? d : c;
  return (e & 4) ? h : l;
}

// A thread's finds wait in two registers and are pushed when the sweep is over, a reservation per warp: the round trip to the
// list's counter (in block 0) is paid once instead of once per find.
struct FoundKeys {
  unsigned long long a, b; uint32_t n, counter; ClusterSmem* s;
  __device__ __forceinline__ void init(ClusterSmem& sm, uint32_t counter_addr) { n = 0u; counter = counter_addr; s = &sm; }
  __device__ __forceinline__ void put(uint32_t slot, unsigned long long key) const {
    if (slot < static_cast<uint32_t>(kCList)) for (int q = 0; q < s->C; q++) cst_u64(cluster_addr(&s->list[slot], q), key);
  }
  __device__ __forceinline__ void add(float z, int idx) {
    const unsigned long long key = (static_cast<unsigned long long>(fkey(canon_zero(z))) << 32) | (0xFFFFFFFFu - static_cast<uint32_t>(idx));
    if (n == 0u) { a = key; n = 1u; } else if (n == 1u) { b = key; n = 2u; } else put(catom_add(counter, 1u), key);
  }
  __device__ __forceinline__ void flush() {                                 // whole warps
    const int lane = threadIdx.x & 31;
    __syncwarp();
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    if (!total) return;
    uint32_t base = 0u;
    if (lane == 0) base = catom_add(counter, total);
    base = __shfl_sync(kFull, base, 0) + incl - n;
    if (n > 0u) put(base, a);
    if (n > 1u) put(base + 1u, b);
  }
};

// The first look at the row: maximum, its lowest index, smallest finite logit, odd values; the group maxima; the slice's copy.
// BF16: a NaN or a magnitude below 2^-39 that is not 0 makes the row odd (one packed test per two logits passes the codes of 2^-39 .. 2^25; a mask
// of -1e9 or the type's lowest value fails it and is looked at closely); binary32: NaN is looked for. +inf shows in the maximum.
template <bool F32, bool CACHED, int B>
static __device__ __noinline__ void phase_load(ClusterSmem& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ClusterRow R = s.R;
  float4* vals = const_cast<float4*>(R.vals);
  float best = -INFINITY, low = INFINITY, glow = INFINITY, gm = -INFINITY;
  int best_c = -1, group = 0;
  bool odd = false;
  const int every = s.every;
  int left = every;
  auto close_group = [&]() { s.gmax[group * B + tid] = gm; if (gm > -INFINITY) glow = fminf(glow, gm); gm = -INFINITY; left = every; group++; };
  {
    int c = R.c0 + tid;
    RawChunk<F32> q;
    if (c < R.c1) q = load_raw<F32>(R, c);
#pragma unroll 1
    for (; c < R.c1;) {
      const int cn = c + B;
      RawChunk<F32> qn = q;
      if (cn < R.c1) qn = load_raw<F32>(R, cn);
      if (F32) {
        const uint4 b = q.a[F32 ? 1 : 0];
        const uint32_t w[8] = {q.a[0].x, q.a[0].y, q.a[0].z, q.a[0].w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 8; e++) odd = odd || (__uint_as_float(w[e]) != __uint_as_float(w[e]));
      } else {
        const uint32_t w[4] = {q.a[0].x, q.a[0].y, q.a[0].z, q.a[0].w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t y = w[k] + 0x14001400u;                            // the window's codes get bits 14:13 = 10 (sample_hist.cuh)
          if ((y & 0x60006000u) != 0x40004000u) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const uint32_t code = h ? w[k] >> 16 : w[k] & 0xFFFFu, mag = code & 0x7FFFu;
              odd = odd || (mag != 0u && mag < 0x2C00u) || mag > 0x7F80u;
            }
          }
        }
      }
      float z[8];
      widen_raw<F32>(R, q, c, z);
      float mx = z[0], mn = z[0];
#pragma unroll
      for (int e = 1; e < 8; e++) { mx = fmaxf(mx, z[e]); mn = fminf(mn, z[e]); }
      if (mn == -INFINITY) {
        mn = INFINITY;
#pragma unroll
        for (int e = 0; e < 8; e++) if (z[e] > -INFINITY) mn = fminf(mn, z[e]);
      }
      low = fminf(low, mn);
      if (mx > best) { best = mx; best_c = c; }
      gm = fmaxf(gm, mx);
      if (--left == 0) close_group();
      if (CACHED) { vals[c - R.c0] = make_float4(z[0], z[1], z[2], z[3]); vals[R.nv + c - R.c0] = make_float4(z[4], z[5], z[6], z[7]); }
      q = qn; c = cn;
    }
    if (left != every) close_group();
  }
  uint64_t mine = 0ull;
  if (best_c >= 0) {                                                        // the lowest index of this thread's maximum
    float z[8];
    if (CACHED) {
      const float4 a = vals[best_c - R.c0], b = vals[R.nv + best_c - R.c0];
      z[0] = a.x; z[1] = a.y; z[2] = a.z; z[3] = a.w; z[4] = b.x; z[5] = b.y; z[6] = b.z; z[7] = b.w;
    } else { const RawChunk<F32> q = load_raw<F32>(R, best_c); widen_raw<F32>(R, q, best_c, z); }
    int at = 0;
#pragma unroll
    for (int e = 7; e >= 0; e--) if (z[e] == best) at = e;
    mine = pack_best(canon_zero(best), static_cast<uint32_t>(8 * best_c + at - R.off));
  }
  const int C = s.C;
  mine = warp_max_u64(mine);
  const uint32_t wl = warp_min_u32(fkey(low)), wg = warp_min_u32(fkey(glow));
  if (lane == 0) { s.scratch[warp] = mine; s.warp_f[warp] = fkey_inv(wl); s.warp_g[warp] = fkey_inv(wg); }
  const int any_odd = __syncthreads_or(odd);
  if (C > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");    // every block of the cluster runs
  if (warp == 0) {
    const uint64_t b = warp_max_u64(lane < B / 32 ? s.scratch[lane] : 0ull);
    const uint32_t l = warp_min_u32(lane < B / 32 ? fkey(s.warp_f[lane]) : 0xFFFFFFFFu), g = warp_min_u32(lane < B / 32 ? fkey(s.warp_g[lane]) : 0xFFFFFFFFu);
    if (lane < C) {
      cst_u64(cluster_addr(&s.x_best[s.rank], lane), b);
      cst_u32(cluster_addr(&s.x_low[s.rank], lane), __float_as_uint(fkey_inv(l)));
      cst_u32(cluster_addr(&s.x_glow[s.rank], lane), __float_as_uint(fkey_inv(g)));
      cst_u32(cluster_addr(&s.x_flags[s.rank], lane), any_odd ? 1u : 0u);
    }
  }
  cluster_sync(C);
  if (warp == 0) {
    const bool have = lane < C;
    const uint64_t top = warp_max_u64(have ? s.x_best[lane] : 0ull);
    const uint32_t l = warp_min_u32(have ? fkey(s.x_low[lane]) : 0xFFFFFFFFu), g = warp_min_u32(have ? fkey(s.x_glow[lane]) : 0xFFFFFFFFu);
    const bool bad = __any_sync(kFull, have && s.x_flags[lane] != 0u) != 0;
    if (lane == 0) {
      const float v = best_value(top);
      s.vmax = v; s.arg = static_cast<int>(best_index(top)); s.vmin = fkey_inv(l); s.gmin = fkey_inv(g);
      s.fallback = bad || top == 0ull || !(fabsf(v) < INFINITY);
    }
  }
  __syncthreads();
}

// The bins of this block's slice.
template <bool F32, bool CACHED>
static __device__ __noinline__ void sweep_bins(ClusterSmem& s, uint32_t kinds) {   // kinds: 1 counts, 2 softmass, 4 draw weights
  const ClusterRow R = s.R;
  const bool use_cnt = kinds & 1u, use_m = kinds & 2u, use_w = kinds & 4u;
  const double inv_t = s.inv_t, vmax64 = static_cast<double>(s.vmax);
  const ClusterBins bins{s.vmax, s.scale, s.window};
  const float vmax = s.vmax, c2 = s.c2;
  if (bins.window != -1) {                                                  // (rare: a bin that more logits share than a list holds)
    sweep<F32, CACHED>(R, [&](int, const float (&z)[8]) {
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const uint32_t b = bins.of(z[e]);
        if (b >= static_cast<uint32_t>(kCBins) || !(z[e] > -INFINITY)) continue;
        atomicAdd(&s.cnt[b], 1u);
        if (use_w) bin_add_u64(s.lo[1], s.hi[1], b, weight_q40(z[e], vmax, c2));
        if (use_m) bin_add_u64(s.lo[0], s.hi[0], b, fixed43(exp64((static_cast<double>(z[e]) - vmax64) * inv_t, s.exp_tab)));
      }
    });
    return;
  }
  if (use_m) {
    // a logit's exp is its bin centre's times a short polynomial: |z - centre| / T <= 31 / 2046, the remainder of degree 4 is below 7e-12
    const double a2 = 0.5 * inv_t * inv_t, a3 = a2 * inv_t * (1.0 / 3.0), a4 = a3 * inv_t * 0.25;
    // (Its distance below the maximum is the bin's number times the bins' width: kept beside the exp it made the look-ups at random bins 16 bytes
    // wide: 14.1 us so, 13.2 without, for 38 K binary32 logits a block.)
    const double step = 1.0 / static_cast<double>(s.scale);
    const float deep = 31.0f * s.T;                                         // logits this far below the maximum: their fixed-point softmass is 0
    sweep<F32, CACHED>(R, [&](int, const float (&z)[8]) {
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        uint32_t b[4]; uint64_t m[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float v = z[h + e];
          b[e] = bins.coarse(v);
          const double bin = __dsub_rn(__hiloint2double(0x43300000, static_cast<int>(b[e])), 4503599627370496.0);   // (2^52 + b) - 2^52
          const double d = __fma_rn(bin, step, static_cast<double>(v) - vmax64);
          m[e] = fixed43(s.bin_exp[b[e]] * __fma_rn(__fma_rn(__fma_rn(__fma_rn(a4, d, a3), d, a2), d, inv_t), d, 1.0));
          if (!(vmax - v < deep)) m[e] = 0ull;                              // (also -inf, whose polynomial means nothing)
        }
        if (use_cnt) {
#pragma unroll
          for (int e = 0; e < 4; e++) if (z[h + e] > -INFINITY) atomicAdd(&s.cnt[b[e]], 1u);
        }
        if (use_w) {
          uint64_t w[4];
          weight_q40_x2(z[h], z[h + 1], vmax, c2, w[0], w[1]);
          weight_q40_x2(z[h + 2], z[h + 3], vmax, c2, w[2], w[3]);
          bin_add4_u64(s.lo[1], s.hi[1], b, w);
        }
        bin_add4_u64(s.lo[0], s.hi[0], b, m);
      }
    });
    return;
  }
  sweep<F32, CACHED>(R, [&](int, const float (&z)[8]) {
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      uint32_t b[4];
#pragma unroll
      for (int e = 0; e < 4; e++) b[e] = bins.coarse(z[h + e]);
      if (use_cnt) {
#pragma unroll
        for (int e = 0; e < 4; e++) if (z[h + e] > -INFINITY) atomicAdd(&s.cnt[b[e]], 1u);
      }
      if (use_w) {
        uint64_t w[4];
        weight_q40_x2(z[h], z[h + 1], vmax, c2, w[0], w[1]);                // (-inf: weight 0)
        weight_q40_x2(z[h + 2], z[h + 3], vmax, c2, w[2], w[3]);
        bin_add4_u64(s.lo[1], s.hi[1], b, w);
      }
    }
  });
}

// Fills the bins of the slices, adds them up over the cluster, and forms their running sums. dirty: something has lain over the bins.
template <bool F32, bool CACHED, int B>
static __device__ __noinline__ void phase_bins(ClusterSmem& s, uint32_t kinds, bool dirty) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = s.C, rank = s.rank;
  const bool use_cnt = kinds & 1u, use_m = kinds & 2u, use_w = kinds & 4u;
  if (dirty) {
    cluster_sync(C);                                                        // (the lists that lie over the bins are no longer read)
    for (int i = tid; i < kCBins; i += B) { s.cnt[i] = 0u; s.lo[0][i] = 0u; s.lo[1][i] = 0u; s.hi[0][i] = 0u; s.hi[1][i] = 0u; }
  }
  if (use_m && s.window == -1) {
    const double step = 1.0 / static_cast<double>(s.scale);
    for (int b = tid; b < kCBins; b += B) s.bin_exp[b] = exp64(-(static_cast<double>(b) * step) * s.inv_t, s.exp_tab);
  }
  __syncthreads();
  sweep_bins<F32, CACHED>(s, kinds);
  cluster_sync(C);
  // a share of the bins each: a warp adds up 32 neighbouring bins of one block after the other, then pushes the totals to all
  const int share = kCBins / C;
  if (C == 1) {
    for (int b = tid; b < kCBins; b += B) {
      if (use_cnt) s.r_cnt[b] = s.cnt[b];
      if (use_m) s.r_sum[0][b] = s.lo[0][b] + (static_cast<unsigned long long>(s.hi[0][b]) << 32);
      if (use_w) s.r_sum[1][b] = s.lo[1][b] + (static_cast<unsigned long long>(s.hi[1][b]) << 32);
    }
  } else {
    const int strips = share / 32;
    // unit = (strip of 32 bins, which sum): counts 0, softmass 1, weights 2
    const int units = strips * 3;
    for (int un = warp; un < units; un += B / 32) {
      const int kind = un / strips, bin = rank * share + (un - kind * strips) * 32 + lane;
      if (!((kinds >> kind) & 1u)) continue;                            // warp-uniform
      if (kind == 0) {
        uint32_t v[kCMaxRanks], n = 0u;
#pragma unroll
        for (int q = 0; q < kCMaxRanks; q++) v[q] = q < C ? cld_u32(cluster_addr(&s.cnt[bin], q)) : 0u;
#pragma unroll
        for (int q = 0; q < kCMaxRanks; q++) n += v[q];
        for (int q = 0; q < C; q++) cst_u32(cluster_addr(&s.r_cnt[bin], q), n);
      } else {
        const uint32_t *lo = s.lo[kind - 1], *hi = s.hi[kind - 1];
        unsigned long long m = 0ull;
#pragma unroll
        for (int h = 0; h < kCMaxRanks; h += 8) {
          uint32_t a[8], b[8];
#pragma unroll
          for (int q = 0; q < 8; q++) { a[q] = h + q < C ? cld_u32(cluster_addr(&lo[bin], h + q)) : 0u; b[q] = h + q < C ? cld_u32(cluster_addr(&hi[bin], h + q)) : 0u; }
#pragma unroll
          for (int q = 0; q < 8; q++) m += a[q] + (static_cast<unsigned long long>(b[q]) << 32);
        }
        for (int q = 0; q < C; q++) cst_u64(cluster_addr(&s.r_sum[kind - 1][bin], q), m);
      }
    }
  }
  cluster_sync(C);
  if (use_cnt) scan_counts<B>(s.r_cnt, s.scratch);
  if (use_m) scan_bins<B>(s.r_sum[0], s.scratch);
  if (use_w) scan_bins<B>(s.r_sum[1], s.scratch);
}

// no logit with bin <= b lies below this (the rounding of the bin's arithmetic is 3 units in the last place of the depth)
__device__ __forceinline__ float floor_of_bin(float vmax, float b, float scale) {
  const float d = (b + 0.5f) / scale * (1.0f + 1e-6f);
  return (vmax - d) - (fabsf(vmax) + d) * 4e-7f;
}
// ... and none with bin >= b above this
__device__ __forceinline__ float ceil_of_bin(float vmax, float b, float scale) {
  const float d = (b - 0.5f) / scale * (1.0f - 1e-6f);
  return (vmax - d) + (fabsf(vmax) + d) * 4e-7f;
}

// A list: its counter is one of two words of block 0, used in turn (the other one is cleared meanwhile). again: a list came before it.
__device__ __forceinline__ uint32_t begin_list(ClusterSmem& s, int turn) {
  if (turn > 0) cluster_sync(s.C);                                          // nobody reads the previous list any more
  if (threadIdx.x == 0) s.list_n[(turn & 1) ^ 1] = 0u;
  return cluster_addr(&s.list_n[turn & 1], 0);
}
__device__ __forceinline__ int end_list(ClusterSmem& s, uint32_t counter) {
  cluster_sync(s.C);
  return static_cast<int>(cld_u32(counter));
}

// The logits of bin b as an ordered list; returns how many (> kCList: no list). They are looked at closely only between two values
// that no logit of the (coarse) bin can lie outside of.
template <bool F32, bool CACHED, int B>
static __device__ __noinline__ int phase_bin_list(ClusterSmem& s, uint32_t b, int turn) {
  const ClusterBins bins{s.vmax, s.scale, s.window};
  float zl, zh;
  if (bins.window == kLogBins || bins.window >= kCBins) {                    // (the depth's rounding is half a unit in its last place)
    const uint32_t lb = bins.window == kLogBins ? b : static_cast<uint32_t>(bins.window - kCBins);
    const float near = log_bin_edge(lb), far = log_bin_edge(lb + 1u);
    zl = far == INFINITY ? -FLT_MAX : (bins.vmax - far) - (fabsf(bins.vmax) + far) * 4e-7f;
    zh = fminf((bins.vmax - near) + (fabsf(bins.vmax) + near) * 4e-7f, bins.vmax);
  } else {
    const uint32_t cb = bins.window < 0 ? b : static_cast<uint32_t>(bins.window);
    zl = cb >= static_cast<uint32_t>(kCBins - 1) ? -FLT_MAX : floor_of_bin(bins.vmax, static_cast<float>(cb), bins.scale);
    zh = cb > 0u ? ceil_of_bin(bins.vmax, static_cast<float>(cb), bins.scale) : bins.vmax;
  }
  FoundKeys found;
  found.init(s, begin_list(s, turn));
  {
    const ClusterRow R = s.R;
    sweep<F32, CACHED>(R, [&](int c, const float (&z)[8]) {
      uint32_t m = 0u;
#pragma unroll
      for (int e = 0; e < 8; e++) m |= (z[e] >= zl && z[e] <= zh) ? 1u << e : 0u;
#pragma unroll 1
      for (; m; m &= m - 1u) {                                              // usually one
        const int e = __ffs(static_cast<int>(m)) - 1;
        const float v = pick8(z, e);
        if (bins.of(v) == b) found.add(v, 8 * c + e - R.off);
      }
    });
  }
  found.flush();
  const int n = end_list(s, found.counter);
  // Neighbouring BF16 values of magnitude >= a lie a / 256 apart or more: four of the list's bins, where its span is no more than a. The order of equal ones
  // matters to the draw by inverse CDF alone.
  const float least = zl > 0.0f ? zl : zh < 0.0f ? -zh : 0.0f;
  const bool in_bins = !F32 && s.R.pen == nullptr && !s.inverse && zh - zl <= least;
  if (n <= kCList) order_list<B>(s, n, zh, fmaxf(zl, s.vmin), in_bins, F32 || in_bins ? kCRankOrder : kCRankOrderFew);   // (few values, penalised or not)
  return n;
}

// Every logit >= zf (and above -inf) into the list; the row's FP32 mass into x_mass when asked for. Returns the list's length.
template <bool F32, bool CACHED>
static __device__ __noinline__ int phase_select(ClusterSmem& s, float zf, bool need_z) {
  const float c2a = static_cast<float>(1.4426950408889634 * s.inv_t), nb = __fmul_rn(-s.vmax, c2a);
  FoundKeys found;
  found.init(s, begin_list(s, 0));
  float2 acc = make_float2(0.0f, 0.0f);
  {
    const ClusterRow R = s.R;
    sweep<F32, CACHED>(R, [&](int c, const float (&z)[8]) {
      const float mx = fmaxf(fmaxf(fmaxf(z[0], z[1]), fmaxf(z[2], z[3])), fmaxf(fmaxf(z[4], z[5]), fmaxf(z[6], z[7])));
      if (need_z) {                                                         // (two at a time, a chunk's terms added up before they join the thread's sum)
        float2 t[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float2 x = __ffma2_rn(make_float2(z[2 * k], z[2 * k + 1]), make_float2(c2a, c2a), make_float2(nb, nb));
          t[k] = make_float2(ex2_approx(x.x), ex2_approx(x.y));
        }
        acc = __fadd2_rn(acc, __fadd2_rn(__fadd2_rn(t[0], t[1]), __fadd2_rn(t[2], t[3])));
      }
      if (mx >= zf) {
        uint32_t m = 0u;
#pragma unroll
        for (int e = 0; e < 8; e++) m |= (z[e] >= zf && z[e] > -INFINITY) ? 1u << e : 0u;
#pragma unroll 1
        for (; m; m &= m - 1u) { const int e = __ffs(static_cast<int>(m)) - 1; found.add(pick8(z, e), 8 * c + e - R.off); }
      }
    });
  }
  found.flush();
  if (need_z) {
    // the common factor that nb's rounding leaves is taken out exactly
    const double m = cblock_sum_f64(static_cast<double>(acc.x) + static_cast<double>(acc.y), s.scratch) * exp2(-(static_cast<double>(s.vmax) * static_cast<double>(c2a) + static_cast<double>(nb)));
    if (static_cast<int>(threadIdx.x) < s.C) cst_u64(cluster_addr(&s.x_mass[s.rank], threadIdx.x), __double_as_longlong(m));
  }
  return end_list(s, found.counter);
}

// The FP64 softmass of the row's logits >= tau, the same in every block. `slots`: where the blocks' shares meet.
template <bool F32, bool CACHED>
static __device__ __noinline__ double phase_mass64(ClusterSmem& s, float tau, double* slots) {
  const double inv_t = s.inv_t, vmax64 = static_cast<double>(s.vmax);
  double m = 0.0;
  {
    const ClusterRow R = s.R;
    sweep<F32, CACHED>(R, [&](int, const float (&z)[8]) {
#pragma unroll
      for (int e = 0; e < 8; e++) if (z[e] >= tau && z[e] > -INFINITY) m += exp64((static_cast<double>(z[e]) - vmax64) * inv_t, s.exp_tab);
    });
  }
  m = cblock_sum_f64(m, s.scratch);
  if (static_cast<int>(threadIdx.x) < s.C) cst_u64(cluster_addr(&slots[s.rank], threadIdx.x), __double_as_longlong(m));
  cluster_sync(s.C);
  double total = 0.0;
  for (int q = 0; q < s.C; q++) total += slots[q];
  return total;
}

// The Gumbel-max draw over the logits >= tau. The kept logits of a warp wait in a queue: a hash is the cost here, and no lane idles
// at one.
template <bool F32, bool CACHED, int B>
static __device__ __noinline__ void phase_gumbel(ClusterSmem& s, float tau) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  GumbelScan g;
  // the key of the maximum: a start that most logits cannot reach
  g.init(s.seed, s.step, s.t_id, s.T, __fadd_rn(__fmul_rn(s.vmax, __double2float_rn(s.inv_t)), gumbel(s.seed, s.step, s.t_id, static_cast<uint32_t>(s.arg))));
  __syncthreads();                                                          // (the queues lie over the lists)
  {
    const ClusterRow R = s.R;
    float2* queue = s.queue[warp];
    int waiting = 0, c = R.c0 + tid;
    RawChunk<F32> ahead;
    if (!CACHED && c < R.c1) ahead = load_raw<F32>(R, c);
#pragma unroll 1
    for (; c - lane < R.c1; c += B) {                                       // whole warps: lanes beyond the slice hold -inf
      float z[8];
      if (c < R.c1) {
        if (CACHED) {
          const float4 a = R.vals[c - R.c0], b = R.vals[R.nv + c - R.c0];
          z[0] = a.x; z[1] = a.y; z[2] = a.z; z[3] = a.w; z[4] = b.x; z[5] = b.y; z[6] = b.z; z[7] = b.w;
        } else {
          const RawChunk<F32> q = ahead;
          if (c + B < R.c1) ahead = load_raw<F32>(R, c + B);
          widen_raw<F32>(R, q, c, z);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; e++) z[e] = -INFINITY;
      }
      uint32_t votes[8];
#pragma unroll
      for (int e = 0; e < 8; e++) votes[e] = __ballot_sync(kFull, z[e] >= tau && z[e] > -INFINITY);
#pragma unroll
      for (int e = 0; e < 8; e++) {
        if ((votes[e] >> lane) & 1u) queue[waiting + __popc(votes[e] & ((1u << lane) - 1u))] = make_float2(canon_zero(z[e]), __uint_as_float(static_cast<uint32_t>(8 * c + e - R.off)));
        waiting += __popc(votes[e]);
        if ((e & 1) && waiting >= 64) {                                     // (at most 63 + 64 wait) two keys per lane, from the queue's end
          __syncwarp();
          const float2 a = queue[waiting - 64 + lane], b = queue[waiting - 32 + lane];
          __syncwarp();
          waiting -= 64;
          g.offer2(a.x, __float_as_uint(a.y), b.x, __float_as_uint(b.y));
        }
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < waiting; i += 32) g.offer2(queue[i].x, __float_as_uint(queue[i].y), -INFINITY, 0u);
    __syncwarp();
  }
  const uint64_t win_b = cblock_max_u64(g.best, s.scratch);
  const float rival = (g.best == win_b) ? g.second : (g.best ? best_value(g.best) : -INFINITY);
  const uint32_t rk = warp_max_u32(fkey(rival));
  if (lane == 0) s.warp_f[warp] = fkey_inv(rk);
  __syncthreads();
  if (warp == 0) {
    const uint32_t r = warp_max_u32(lane < B / 32 ? fkey(s.warp_f[lane]) : 0u);
    if (lane < s.C) {
      cst_u64(cluster_addr(&s.x_key[s.rank], lane), win_b);
      cst_u32(cluster_addr(&s.x_rival[s.rank], lane), __float_as_uint(fkey_inv(r)));
    }
  }
  cluster_sync(s.C);
  if (warp == 0) {
    const uint64_t key = lane < s.C ? s.x_key[lane] : 0ull;
    const uint64_t win = warp_max_u64(key);
    if (win) {
      const float edge = best_value(win) - 4e-6f;
      const bool tie = (lane < s.C && s.x_rival[lane] >= edge) || (key && key != win && best_value(key) >= edge);
      const bool any = __any_sync(kFull, tie) != 0;
      if (lane == 0) { s.o_token = static_cast<int>(best_index(win)); if (any) s.o_status |= LM_STATUS_NEAR_TIE; }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ float list_value(const ClusterSmem& s, int i) { return fkey_inv(static_cast<uint32_t>(s.sorted[i] >> 32)); }
__device__ __forceinline__ int list_index(const ClusterSmem& s, int i) { return static_cast<int>(0xFFFFFFFFu - static_cast<uint32_t>(s.sorted[i])); }
// The weight of the ordered list's entries at or above tau.
static __device__ __noinline__ uint64_t list_weight(ClusterSmem& s, int n, float tau) {
  uint64_t w = 0ull;
  for (int i = threadIdx.x; i < n; i += blockDim.x) if (list_value(s, i) >= tau) w += weight_q40(list_value(s, i), s.vmax, s.c2);
  return cblock_sum_u64(w, s.scratch);
}
// The draw by inverse CDF inside the ordered list (n entries; those at or above tau are kept): `base` = the kept weight above it.
static __device__ __noinline__ void pick_in_list(ClusterSmem& s, int n, float tau, uint64_t base, uint64_t target) {
  uint64_t run = base;
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += blockDim.x) {                              // uniform trip count
    const int i = i0 + static_cast<int>(threadIdx.x);
    const uint64_t w = (i < n && list_value(s, i) >= tau) ? weight_q40(list_value(s, i), s.vmax, s.c2) : 0ull;
    uint64_t tot = 0ull;
    const uint64_t before = run + cblock_scan_u64(w, s.scratch, &tot);
    if (w && before <= target && target < before + w) s.o_token = list_index(s, i);
    run += tot;
    __syncthreads();
  }
}

// The group maxima counted in bins of their depth below the row's maximum (16-bit counts pushed to every block, added up there): the bin of the
// top_k-th of them (-1: there are fewer), and how many lie down to that bin, the bin included. kExponent: bins by the depth's exponent and one bit.
template <bool kExponent, int B>
__device__ __forceinline__ int bound_of_maxima(ClusterSmem& s, float mscale, uint32_t* through) {
  const int tid = threadIdx.x, lane = tid & 31, C = s.C;
  const float vmax = s.vmax;
  {
    const ClusterBins mb{vmax, mscale, -1};
    const int mine = (s.R.c1 - s.R.c0 - tid + B - 1) / B, groups = (mine + s.every - 1) / s.every;   // (mine may be negative: no group)
    for (int g = 0; g < groups; g++) {
      const float m = s.gmax[g * B + tid];
      if (m > -INFINITY) atomicAdd(&s.max_cnt[kExponent ? __float_as_uint(__fsub_rn(vmax, m)) >> 22 : min(mb.coarse(m), static_cast<uint32_t>(kCMaxBins - 1))], 1u);
    }
  }
  __syncthreads();
  for (int i = tid; i < C * (kCMaxBins / 2); i += B) {                     // (at most 4096 groups a block: 16 bits)
    const int q = i / (kCMaxBins / 2), w = i - q * (kCMaxBins / 2);
    cst_u32(cluster_addr(&s.x_max[s.rank][w], q), s.max_cnt[2 * w] | (s.max_cnt[2 * w + 1] << 16));
  }
  cluster_sync(C);
  if (tid < kCMaxBins / 2) {
    uint32_t n0 = 0u, n1 = 0u;
    for (int q = 0; q < C; q++) { const uint32_t w = s.x_max[q][tid]; n0 += w & 0xFFFFu; n1 += w >> 16; }
    s.totals[2 * tid] = n0; s.totals[2 * tid + 1] = n1;
  }
  __syncthreads();
  // every warp for itself: lane l holds 16 bins
  uint32_t v[kCMaxBins / 32], sum = 0u;
#pragma unroll
  for (int j = 0; j < kCMaxBins / 32; j += 4) {
    const uint4 q = *reinterpret_cast<const uint4*>(&s.totals[lane * (kCMaxBins / 32) + j]);
    v[j] = q.x; v[j + 1] = q.y; v[j + 2] = q.z; v[j + 3] = q.w; sum += q.x + q.y + q.z + q.w;
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
  const uint32_t k = static_cast<uint32_t>(s.top_k);
  uint32_t run = incl - sum, reached = 0u; int at = -1;
#pragma unroll
  for (int j = 0; j < kCMaxBins / 32; j++) { run += v[j]; if (at < 0 && run >= k) { at = lane * (kCMaxBins / 32) + j; reached = run; } }
  const uint32_t hits = __ballot_sync(kFull, at >= 0);
  if (!hits) return -1;
  *through = __shfl_sync(kFull, reached, __ffs(hits) - 1);
  return __shfl_sync(kFull, at, __ffs(hits) - 1);
}

// The bound again where something far below the rest (a group of nothing but masked logits) has stretched the linear bins until the bin of the
// top_k-th holds far more than top_k: bins by exponent find the range that matters, linear ones divide that. (4 rows of 151,936, a third at
// -1e4, top_k 50: 63 us by the search that an overflowing list leads to, 25 us so; without a mask 19.)
template <int B>
static __device__ __noinline__ int narrower_bound(ClusterSmem& s, float* mscale) {
  auto again = [&]() {
    cluster_sync(s.C);                                                      // (the counts of the pass before are no longer read)
    for (int i = threadIdx.x; i < kCMaxBins; i += B) s.max_cnt[i] = 0u;
    __syncthreads();
  };
  uint32_t through;
  again();
  const int e = bound_of_maxima<true, B>(s, 0.0f, &through);
  // (the top_k-th lies above the lower edge of its bin by exponent: in the first 511 of the linear bins down to that edge)
  *mscale = fminf(static_cast<float>(kCMaxBins - 2) / __uint_as_float(static_cast<uint32_t>(e + 1) << 22), FLT_MAX);
  again();
  return bound_of_maxima<false, B>(s, *mscale, &through);
}

// With a top_k: its whole set as an ordered list, then everything on the list. Returns false when there is no such list.
// *written: the outputs are written (the caller has nothing left to do).
template <bool F32, bool CACHED, int B>
static __device__ __noinline__ bool phase_top_k(ClusterSmem& s, const SampleDev& P, bool* written) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = s.C;
  *written = false;
  // the bound: bins of the group maxima, down to the smallest of them
  const float vmax = s.vmax, gmin = s.gmin;
  float mscale = static_cast<float>(kCMaxBins - 1) / (vmax > gmin ? vmax - gmin : 1.0f);
  uint32_t through = 0u;
  int pick = bound_of_maxima<false, B>(s, mscale, &through);
  if (pick >= 0 && through > 2u * static_cast<uint32_t>(s.top_k) + 64u) pick = narrower_bound<B>(s, &mscale);
  if (pick < 0) return false;                                               // fewer groups than top_k
  // every logit at or above the bound's bin, and (for a top-p over the row) the FP32 mass: one more look at the row. Not at temperatures so
  // small that the rounding of the maximum's exponent is no fraction of a binade (kMassExponent): there the mass is formed in FP64 at once.
  const bool whole = s.has_p && !s.in_topk, need_z = whole && static_cast<double>(fabsf(vmax)) * s.inv_t < kMassExponent;
  const float zf = pick >= kCMaxBins - 1 ? gmin : floor_of_bin(vmax, static_cast<float>(pick), mscale);
  const int n = phase_select<F32, CACHED>(s, zf, need_z);
  if (n > kCList) return false;
  order_list<B>(s, n, vmax, zf);
  const int top_k = s.top_k;
  const float tau_k = top_k <= n ? list_value(s, top_k - 1) : -INFINITY;
  int n_topk = min(top_k, n);                                               // the top-k set (ties kept) is a prefix of the order
  for (bool tied = true; tied;) {                                           // every warp for itself
    const uint32_t v = __ballot_sync(kFull, n_topk + lane < n && list_value(s, n_topk + lane) >= tau_k);
    n_topk += v == kFull ? 32 : __ffs(static_cast<int>(~v)) - 1;
    tied = v == kFull;
  }
  double total = 0.0, err = 0.0;
  if (whole && !need_z) total = phase_mass64<F32, CACHED>(s, -INFINITY, s.x_mass64);
  if (need_z) {
    for (int q = 0; q < C; q++) total += s.x_mass[q];
    const double un = 5.9604644775390625e-8;                                // sample_topk.cuh derives this bound (the reference point here is the maximum itself)
    err = 1.25 * total * (un * (13.9 + 4.0 + static_cast<double>((s.per + B - 1) / B) + 3.0) + 6.6e-7);   // (ln V <= 13.9; a term goes through two additions in its chunk and one a step)
  }
  if (n_topk <= 64 && !s.want_stats) {
    // few candidates: one warp does the rest, with shuffles and votes (vocab_parallel.cuh); rank 0's writes the outputs
    MergeTail t;
    t.key = s.sorted; t.vmax = vmax;
    VpMergeDev M;
    M.flags = s.flags; M.draw = P.draw; M.uniforms = P.uniforms; M.seed = s.seed; M.step = s.step; M.row_offset = P.row_offset;
    M.out_tokens = s.rank == 0 ? P.out_tokens : nullptr; M.out_tau = P.out_tau; M.out_status = P.out_status; M.out_vmax = P.out_vmax; M.out_mass = P.out_mass;
    M.hand_on = 1; M.path_status = s.few ? LM_STATUS_SLICED_PATH : whole && !need_z ? 0u : LM_STATUS_CANDIDATE_PATH;
    *written = true;
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
      if (warp == 0) {
        t.z_total = total; t.amb = 0;
        M.mass_band = total > 0.0 ? err / total : 0.0;
        merge_tail_one_warp<2>(M, s.row, t, n_topk, s.T, top_k, s.top_p, s.min_p, s.inv_t, 0u);
        if (lane == 0) s.amb = t.amb;
      }
      __syncthreads();
      if (!s.amb) break;
      total = phase_mass64<F32, CACHED>(s, -INFINITY, s.x_mass64);          // too close to call in FP32: the row's mass again, in FP64
      err = 0.0;
      if (!s.few) M.path_status = 0u;
    }
    return true;
  }
  // thresholds
  double tau64 = tau_k;
  uint32_t status = s.want_stats || s.few || (whole && !need_z) ? 0u : LM_STATUS_CANDIDATE_PATH;
  if (s.has_p) {
    for (int i = tid; i < n_topk; i += B) s.cum[i] = exp64((static_cast<double>(list_value(s, i)) - static_cast<double>(vmax)) * s.inv_t, s.exp_tab);
    __syncthreads();
    scan_list_f64<B>(s.cum, n_topk, s.warp_d);
    if (s.in_topk) total = s.cum[n_topk - 1];
#pragma unroll 1
    while (true) {
      const double target = static_cast<double>(s.top_p) * total;
      if (tid == 0) { s.hit = kCList; s.hit2 = 0u; }
      __syncthreads();
      for (int i = tid; i < n_topk; i += B) {
        if (i != n_topk - 1 && static_cast<uint32_t>(s.sorted[i + 1] >> 32) == static_cast<uint32_t>(s.sorted[i] >> 32)) continue;
        const double cm = s.cum[i];
        if (cm >= target) atomicMin(&s.hit, static_cast<uint32_t>(i));
        if (err > 0.0 && i < n_topk - 1 && list_value(s, i) > tau_k && fabs(cm - target) <= err) s.hit2 = 1u;
        if (err == 0.0 && fabs(cm - target) <= 1e-12 * total) s.hit2 = 2u;
      }
      __syncthreads();
      const uint32_t hit = s.hit, flag = s.hit2;
      __syncthreads();
      if (flag == 1u) { total = phase_mass64<F32, CACHED>(s, -INFINITY, s.x_mass64); err = 0.0; status &= ~LM_STATUS_CANDIDATE_PATH; continue; }
      if (flag == 2u) status |= LM_STATUS_TOPP_EDGE;
      if (hit < static_cast<uint32_t>(kCList)) { const float tau_p = list_value(s, static_cast<int>(hit)); if (static_cast<double>(tau_p) > tau64) tau64 = tau_p; }
      break;
    }
  }
  if (s.has_m) {
    const double tau_m = static_cast<double>(vmax) + static_cast<double>(s.T) * log(static_cast<double>(s.min_p));
    if (tau_m > tau64) tau64 = tau_m;
  }
  const float tau = __double2float_rn(tau64);
  // the draw
  const uint64_t weight = s.want_w ? list_weight(s, n_topk, tau) : 0ull;
  if (s.want_stats) {                                                       // the kept set lies in the list, and every block holds it
    double m = 0.0;
    for (int i = tid; i < n_topk; i += B) if (list_value(s, i) >= tau) m += exp64((static_cast<double>(list_value(s, i)) - static_cast<double>(vmax)) * s.inv_t, s.exp_tab);
    m = cblock_sum_f64(m, s.scratch);
    if (tid == 0) s.kept_mass = m;
  }
  if (tid == 0) { s.o_tau = tau; s.o_status |= status; s.o_weight = weight; }
  __syncthreads();
  if (s.inverse) {
    if (weight > 0ull) pick_in_list(s, n_topk, tau, 0ull, cdf_target(s.u, weight));
  } else {
    const float inv_t32 = __double2float_rn(s.inv_t);
    uint64_t b1 = 0ull; float second = -INFINITY;
#pragma unroll 1
    for (int i = tid; i < n_topk; i += B) {
      const float v = list_value(s, i);
      if (!(v >= tau)) continue;
      const uint32_t idx = static_cast<uint32_t>(list_index(s, i));
      const float key = __fadd_rn(__fmul_rn(v, inv_t32), gumbel(s.seed, s.step, s.t_id, idx));
      const uint64_t pk = pack_best(key, idx);
      if (pk > b1) { if (b1) second = fmaxf(second, best_value(b1)); b1 = pk; } else second = fmaxf(second, key);
    }
    const uint64_t win = cblock_max_u64(b1, s.scratch);
    if (win) {
      const float rival = (b1 == win) ? second : (b1 ? best_value(b1) : -INFINITY);
      const int tie = __syncthreads_or(rival >= best_value(win) - 4e-6f);
      if (tid == 0) { s.o_token = static_cast<int>(best_index(win)); if (tie) s.o_status |= LM_STATUS_NEAR_TIE; }
    }
    __syncthreads();
  }
  return true;
}

// Without a top_k (or with one whose set the list does not hold): up to four searches, each for the bin where something is crossed: the
// top_k-th logit, the top_p mass, tau (what its own bin keeps), the draw. They are steps of one loop. What a search leaves: the ordered
// logits of its bin in s.sorted[0 .. list_len), and what lies above them. Returns false when the row is not decided here.
template <bool F32, bool CACHED, int B>
static __device__ __noinline__ bool phase_search(ClusterSmem& s, bool dirty) {
  const int tid = threadIdx.x;
  enum { kCount, kMass, kTau, kDraw };
  int list_len = 0, list_tag = -1, turn = dirty ? 1 : 0;
  uint32_t above_n = 0u; uint64_t above_m = 0ull, above_w = 0ull;
  bool fresh = false, have_tau = false;                                     // fresh: the bins are those of the whole row
  int attempt = F32 ? 1 : 0;                                                // BF16: the weights' sums decide most rows (attempt 0)
  double tau64 = -INFINITY, topk_mass = 0.0, target_m = 0.0, err_m = 0.0;
  float tau_k = -INFINITY, tau = -INFINITY;
  uint64_t target_w = 0ull;
  if (tid == 0) {
    // exponents down to 2^-44.7 (below that neither sum has anything); a count alone can cross anywhere
    const float span = s.vmax - s.vmin, range = (s.has_k && !s.has_p && !s.want_w) ? span : fminf(span, 31.0f * s.T);
    s.scale = static_cast<float>(kCBins - 1) / (range > 0.0f ? range : 1.0f);
  }
  int step = s.has_k ? kCount : s.has_p ? kMass : kTau;
#pragma unroll 1
  while (true) {
    const bool use_m = s.has_p && attempt == 1;
    const uint32_t kinds = (s.has_k ? 1u : 0u) | (use_m ? 2u : 0u) | ((s.want_w || (s.has_p && attempt == 0)) ? 4u : 0u);
    const unsigned long long* sums = s.r_sum[use_m ? 0 : 1];                // of the softmass
    const double unit = use_m ? 0x1p-43 : 0x1p-40;
    if (step == kTau) {                                                     // the thresholds are known
      if (s.has_m) {
        const double tau_m = static_cast<double>(s.vmax) + static_cast<double>(s.T) * log(static_cast<double>(s.min_p));
        if (!have_tau || tau_m > tau64) tau64 = tau_m;
        have_tau = true;
      }
      tau = have_tau ? __double2float_rn(tau64) : -INFINITY;
      if (!s.want_w || tau > s.vmax) break;                                 // (a min_p above 1 keeps nothing)
    }
    above_n = 0u; above_m = above_w = 0ull;
    bool refill = !fresh, empty = false, again = false;
    int base = -1;                                                          // the bins of level 0: linear, or (kLogBins) by exponent
#pragma unroll 1
    for (int level = 0;; level++) {
      if (refill) {
        if (level == 0 && tid == 0) s.window = base;                        // (phase_bins has a barrier before it reads this)
        if (level == 0) __syncthreads();
        phase_bins<F32, CACHED, B>(s, kinds | (level ? 1u : 0u), dirty);
        dirty = true; fresh = level == 0 && base == -1; list_tag = -1; refill = false;
      }
      if (level == 0 && step == kMass) {
        const double row_total = static_cast<double>(sums[kCBins - 1]) * unit;
        target_m = static_cast<double>(s.top_p) * ((s.in_topk && tau_k > -INFINITY) ? topk_mass : row_total);
        const double n = static_cast<double>(s.R.V);
        err_m = use_m ? 1.25 * n * 0x1p-44 + kCMassBand * row_total : row_total * weight_band(s.R.V) + 1.25 * n * 0x1p-40;
      }
      // the bin
      uint32_t b;
      if (step == kTau) {
        const ClusterBins bins{s.vmax, s.scale, s.window};
        b = tau > -INFINITY ? bins.of(tau) : kCBins;
        // a bin in which nothing weighs anything (or no bin: nothing is cut off) leaves nothing to order
        if (b >= static_cast<uint32_t>(kCBins) || s.r_sum[1][b] == (b ? s.r_sum[1][b - 1] : 0ull)) {
          above_w += tau > -INFINITY ? (b < static_cast<uint32_t>(kCBins) ? s.r_sum[1][b] : 0ull) : s.r_sum[1][kCBins - 1];
          empty = true; break;
        }
      } else {
        if (tid == 0) s.pick = kCBins;
        __syncthreads();
        for (int i = tid; i < kCBins; i += B) {
          const bool reached = step == kCount ? above_n + s.r_cnt[i + 1] >= static_cast<uint32_t>(s.top_k)
                             : step == kMass ? static_cast<double>((use_m ? above_m : above_w) + sums[i]) * unit >= target_m : above_w + s.r_sum[1][i] > target_w;
          if (reached) { atomicMin(&s.pick, static_cast<uint32_t>(i)); break; }
        }
        __syncthreads();
        b = s.pick;
        if (b >= static_cast<uint32_t>(kCBins)) { empty = true; break; }
      }
      // with the counts at hand a list that could not hold the bin is not begun
      const uint32_t in_bin = (kinds & 1u) || level ? s.r_cnt[b + 1] - s.r_cnt[b] : 0u;
      // A count can cross where the linear bins do not tell: beyond their range (which is that of the weights), or so near the maximum that a
      // masked logit has stretched them over everything else. The bins by exponent do.
      if (step == kCount && level == 0 && base == -1 && in_bin > static_cast<uint32_t>(kCList) && (b < 4u || b == static_cast<uint32_t>(kCBins - 1))) {
        base = kLogBins; level = -1; refill = true;
        continue;
      }
      if ((kinds & 1u) || level) above_n += s.r_cnt[b];
      if (b && (kinds & 2u)) above_m += s.r_sum[0][b - 1];
      if (b && (kinds & 4u)) above_w += s.r_sum[1][b - 1];
      if (level == 0 && list_tag == static_cast<int>(b)) break;             // the list in hand
      list_len = static_cast<int>(in_bin);
      if (in_bin <= static_cast<uint32_t>(kCList)) {
        list_len = phase_bin_list<F32, CACHED, B>(s, b, turn);
        turn = (turn & 1) ? 2 : 1;                                          // (> 0: a list has come before)
      }
      if (list_len <= kCList) { list_tag = level || base != -1 ? -1 : static_cast<int>(b); break; }
      if (level == 1) return false;                                         // more equal logits than a list holds
      fresh = false; refill = true;
      __syncthreads();                                                      // (where no list was begun, a warp may still be looking tau's bin up with the window as it was)
      if (tid == 0) s.window = base == -1 ? static_cast<int>(b) : kCBins + static_cast<int>(b);
      __syncthreads();
    }
    if (empty) { list_len = 0; list_tag = -1; }
    if (step == kCount) {
      have_tau = true;
      if (!empty) { tau_k = list_value(s, s.top_k - 1 - static_cast<int>(above_n)); tau64 = tau_k; }   // (empty: fewer logits above -inf than top_k)
      if (s.in_topk && s.has_p) {                                           // the mass of the top-k set
        double m = 0.0;
        for (int i = tid; i < list_len; i += B) if (list_value(s, i) >= tau_k) m += exp64((static_cast<double>(list_value(s, i)) - static_cast<double>(s.vmax)) * s.inv_t, s.exp_tab);
        topk_mass = cblock_sum_f64(m, s.scratch) + static_cast<double>(use_m ? above_m : above_w) * unit;
      }
      step = s.has_p ? kMass : kTau;
    } else if (step == kMass) {
      const uint64_t above = use_m ? above_m : above_w;
      const double base = static_cast<double>(above) * unit;
      again = empty || list_len == 0 || (above != 0ull && fabs(base - target_m) <= err_m);
      if (!again) {
        for (int i = tid; i < list_len; i += B) s.cum[i] = exp64((static_cast<double>(list_value(s, i)) - static_cast<double>(s.vmax)) * s.inv_t, s.exp_tab);
        if (tid == 0) { s.hit = kCList; s.hit2 = 0u; }
        __syncthreads();
        scan_list_f64<B>(s.cum, list_len, s.warp_d);
        for (int i = tid; i < list_len; i += B) {
          if (i != list_len - 1 && static_cast<uint32_t>(s.sorted[i + 1] >> 32) == static_cast<uint32_t>(s.sorted[i] >> 32)) continue;
          const double cm = base + s.cum[i];
          if (cm >= target_m) atomicMin(&s.hit, static_cast<uint32_t>(i));
          if (fabs(cm - target_m) <= err_m) s.hit2 = 1u;
        }
        __syncthreads();
        const uint32_t hit = s.hit;
        again = s.hit2 != 0u || hit >= static_cast<uint32_t>(kCList);
        __syncthreads();
        if (!again) {
          const float tau_p = list_value(s, static_cast<int>(hit));
          if (!have_tau || static_cast<double>(tau_p) > tau64) tau64 = tau_p;
          have_tau = true;
        }
      }
      if (!again) step = kTau;
      else if (attempt == 1) return false;
      else { attempt = 1; fresh = false; tau64 = -INFINITY; have_tau = false; tau_k = -INFINITY; step = s.has_k ? kCount : kMass; }   // the finer sums
    } else if (step == kTau) {
      const uint64_t weight = above_w + (list_len ? list_weight(s, list_len, tau) : 0ull);
      if (tid == 0) s.o_weight = weight;
      if (!s.inverse || weight == 0ull) break;
      target_w = cdf_target(s.u, weight);
      if (list_len && target_w >= above_w) { pick_in_list(s, list_len, tau, above_w, target_w); break; }
      step = kDraw;
    } else {
      pick_in_list(s, list_len, tau, above_w, target_w);
      break;
    }
  }
  if (tid == 0) s.o_tau = tau;
  __syncthreads();
  if (!s.inverse && !(tau > s.vmax)) phase_gumbel<F32, CACHED, B>(s, tau);
  return true;
}

// The kept-token probabilities of this block's slice: half a chunk a store where the output is aligned like the row, else element by element (the
// stores of a warp are one line). token >= 0: one-hot. (4 FP32 rows of 151,936 with a top_k, the kept mass from its list included: 21.8 us with a
// sweep for the mass and single elements, 17.9 so.)
template <bool F32, bool CACHED>
static __device__ __noinline__ void phase_probs(const ClusterSmem& s, const SampleDev& P, int token, double inv_mass) {
  const ClusterRow R = s.R;
  float* pr = P.out_probs + static_cast<int64_t>(s.row) * P.probs_stride;
  const int i0 = max(0, 8 * R.c0 - R.off), i1 = min(R.V, 8 * R.c1 - R.off);
  const float tau = s.o_tau;
  const double inv_t = s.inv_t, vmax64 = static_cast<double>(s.vmax);
  if (CACHED && token < 0 && (reinterpret_cast<uintptr_t>(pr - R.off) & 15u) == 0) {
    for (int h = 2 * R.c0 + static_cast<int>(threadIdx.x); h < 2 * R.c1; h += blockDim.x) {
      const float4 v = R.vals[((h & 1) ? R.nv : 0) + ((h >> 1) - R.c0)];
      const float z[4] = {v.x, v.y, v.z, v.w};
      float p[4];
#pragma unroll
      for (int e = 0; e < 4; e++) p[e] = 0.0f;
      if (fmaxf(fmaxf(z[0], z[1]), fmaxf(z[2], z[3])) >= tau) {
#pragma unroll
        for (int e = 0; e < 4; e++) if (z[e] >= tau && z[e] > -INFINITY) p[e] = static_cast<float>(exp64((static_cast<double>(z[e]) - vmax64) * inv_t, s.exp_tab) * inv_mass);
      }
      const int i = 4 * h - R.off;
      if (i >= 0 && i + 4 <= R.V) *reinterpret_cast<float4*>(pr + i) = make_float4(p[0], p[1], p[2], p[3]);
      else for (int e = 0; e < 4; e++) if (i + e >= 0 && i + e < R.V) pr[i + e] = p[e];
    }
    return;
  }
  for (int i = i0 + static_cast<int>(threadIdx.x); i < i1; i += blockDim.x) {
    if (token >= 0) { pr[i] = i == token ? 1.0f : 0.0f; continue; }
    const int j = i + R.off, c = j >> 3, e = j & 7;
    float z;
    if (CACHED) z = reinterpret_cast<const float*>(R.vals + (e < 4 ? 0 : R.nv) + (c - R.c0))[e & 3];
    else {
      z = F32 ? __ldg(reinterpret_cast<const float*>(R.row) + i) : __uint_as_float(static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(R.row) + i)) << 16);
      if (R.pen && ((R.pen[c - R.c0] >> e) & 1u)) z = penalise(z, R.rho, R.pi);
    }
    pr[i] = (z >= tau && z > -INFINITY) ? static_cast<float>(exp64((static_cast<double>(z) - vmax64) * inv_t, s.exp_tab) * inv_mass) : 0.0f;
  }
}

// The row that cluster `at` takes when there are more clusters than run at once: the long rows (no list of a top_k) first, then those with a
// large top_k, so that no long one is begun when the rest are done. At most kOrderRows rows. (64 FP32 rows of 151,936 with mixed knobs, four blocks
// each and one to an SM: 93.8 us in the order of the batch, 72.9 so; 48 BF16 rows of 50,257 53.0 and 47.0; 300 FP32 rows of 50,257 131 and 120.)
template <int B>
static __device__ __noinline__ int row_in_order(const SampleDev& P, int rows, int at, ClusterSmem& s) {
  const int tid = threadIdx.x, lane = tid & 31;
  constexpr int kGroups = kOrderRows / 32;
  uint32_t* count = s.r_cnt;                                                // [2][rows / 32]: the first two kinds per 32 rows
  // (No barrier lies between the kernel's clearing of its bins and the first count: the counts have to be other words, and these are written again
  // before anything else reads them.)
  static_assert(2 * kGroups <= kCBins && offsetof(ClusterSmem, r_cnt) >= offsetof(ClusterSmem, max_cnt) + sizeof(ClusterSmem::max_cnt) &&
                offsetof(ClusterSmem, r_cnt) >= offsetof(ClusterSmem, hi) + sizeof(ClusterSmem::hi), "the counts share no word with what the kernel clears first");
  auto kind_of = [&](int r) {
    if (r >= rows) return 3;
    const int k = P.top_k[r];
    const float T = P.temperature ? P.temperature[r] : P.temperature_s;
    return !(T > 0.0f) ? 2 : (k <= 0 || k > kCListK || (P.flags & LM_FLAG_EXACT_ONLY)) ? 0 : k > 64 ? 1 : 2;
  };
  constexpr int kMine = (kOrderRows + B - 1) / B;
  uint32_t kinds = 0u;                                                      // two bits for each of this thread's rows
#pragma unroll
  for (int m = 0; m < kMine; m++) {
    const int r = tid + m * B;
    if (r - lane >= rows) break;                                            // (warp-uniform)
    const int kind = kind_of(r);
    kinds |= static_cast<uint32_t>(kind) << (2 * m);
    const uint32_t a = __ballot_sync(kFull, kind == 0), b = __ballot_sync(kFull, kind == 1);
    if (lane == 0) { count[r >> 5] = __popc(a); count[kGroups + (r >> 5)] = __popc(b); }
  }
  __syncthreads();
  const int groups = (rows + 31) >> 5;
  uint32_t n0 = 0u, n1 = 0u;                                                // every warp for itself
  for (int g = lane; g < groups; g += 32) { n0 += count[g]; n1 += count[kGroups + g]; }
  n0 = warp_sum_u32(n0); n1 = warp_sum_u32(n1);
  for (int r = tid; r - lane < rows; r += B, kinds >>= 2) {
    const int kind = static_cast<int>(kinds & 3u), mine = r >> 5;
    uint32_t b0 = 0u, b1 = 0u;
    for (int g = lane; g < mine; g += 32) { b0 += count[g]; b1 += count[kGroups + g]; }
    b0 = warp_sum_u32(b0); b1 = warp_sum_u32(b1);
    const uint32_t a = __ballot_sync(kFull, kind == 0), b = __ballot_sync(kFull, kind == 1), below = (1u << lane) - 1u;
    const uint32_t p0 = b0 + __popc(a & below), p1 = b1 + __popc(b & below);
    const uint32_t place = kind == 0 ? p0 : kind == 1 ? n0 + p1 : n0 + n1 + static_cast<uint32_t>(r) - p0 - p1;
    if (kind < 3 && place == static_cast<uint32_t>(at)) s.row = r;
  }
  __syncthreads();
  const int row = s.row;
  __syncthreads();                                                          // (the knobs' thread writes s.row again)
  return row;
}

__host__ __device__ inline size_t cluster_smem_head() { return (sizeof(ClusterSmem) + 127) & ~static_cast<size_t>(127); }

// CACHED: the slices of the row fit the blocks' shared memory.
template <bool F32, bool CACHED, int B, int kPerSM>
__global__ void __launch_bounds__(B, kPerSM) sample_cluster_kernel(const __grid_constant__ SampleDev P, int C, uint32_t call) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ClusterSmem& s = *reinterpret_cast<ClusterSmem*>(smem_raw);
  const int tid = threadIdx.x;
  const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0;
  int row = C > 1 ? static_cast<int>(blockIdx.x) / C : static_cast<int>(blockIdx.x);
  // what needs no device memory comes first, beside the kernel in front of this one
  for (int i = tid; i < kCBins; i += B) { s.cnt[i] = 0u; s.lo[0][i] = 0u; s.lo[1][i] = 0u; s.hi[0][i] = 0u; s.hi[1][i] = 0u; }
  for (int i = tid; i < kCMaxBins; i += B) s.max_cnt[i] = 0u;
  if (tid < 64) s.exp_tab[tid] = exp2(static_cast<double>(tid) * 0.015625);
  after_predecessor();
  int rows = P.rows; uint64_t seed = P.seed; uint32_t noise_step = P.step;
  if (P.state) {                                                            // (as apply_step_state)
    StepStateView st{const_cast<uint32_t*>(P.state), P.t_max, P.g};
    const int active = st.done() ? 0 : static_cast<int>(st.t_this_step());
    rows = active < rows ? active : rows; seed = st.seed(); noise_step = st.step();
  }
  if (row >= rows) return;                                                  // (uniform over the cluster)
  if (call & kCallOrdered) row = row_in_order<B>(P, rows, row, s);
  const int V = P.vocab;
  const float T = P.temperature ? P.temperature[row] : P.temperature_s;
  const bool pen_on = P.history != nullptr && P.hist_len > 0;
  if (C > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this block runs: its memory may be written to
  // ---- set-up: this block's slice, the knobs, clear bins, the history's ids inside the slice --------------------------------------------
  const char* rowp = static_cast<const char*>(P.logits) + static_cast<size_t>(row) * static_cast<size_t>(P.row_stride) * (F32 ? 4 : 2);
  const int head = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(rowp) & 15u)) & 15u) / (F32 ? 4 : 2);
  const int off = head ? 8 - head : 0, n_chunks = (V + off + 7) / 8, per = (n_chunks + C - 1) / C;
  const int c0 = min(n_chunks, rank * per), c1 = min(n_chunks, c0 + per);
  uint8_t* pen = smem_raw + cluster_smem_head() + (CACHED ? static_cast<size_t>(per) * 32 : 0);
  if (tid == 0) {
    s.R = ClusterRow{rowp, V, off, c0, c1, reinterpret_cast<const float4*>(smem_raw + cluster_smem_head()), per, pen_on ? pen : nullptr, P.rho, P.pi};
    int top_k = P.top_k ? P.top_k[row] : P.top_k_s;
    const float top_p = P.top_p ? P.top_p[row] : P.top_p_s, min_p = P.min_p ? P.min_p[row] : P.min_p_s;
    s.seed = seed; s.step = noise_step; s.row = row; s.rank = rank; s.C = C; s.per = per; s.flags = P.flags; s.window = -1;
    s.T = T; s.inv_t = T > 0.0f ? 1.0 / static_cast<double>(T) : 0.0; s.c2 = T > 0.0f ? exp2_scale(T) : 0.0f;
    s.top_k = min(top_k, V); s.top_p = top_p; s.min_p = min_p;
    s.has_k = top_k > 0; s.has_p = top_p > 0.0f && top_p < 1.0f; s.has_m = min_p > 0.0f;
    s.in_topk = (P.flags & LM_FLAG_TOPP_IN_TOPK) && top_k > 0;
    s.inverse = P.draw == LM_DRAW_INVERSE_CDF; s.want_w = s.inverse || P.out_mass != nullptr; s.want_stats = P.out_probs != nullptr || P.out_stats != nullptr;
    s.t_id = static_cast<uint32_t>(P.row_offset + row); s.u = (s.inverse && P.uniforms) ? P.uniforms[row] : 0.0f;
    // group maxima (for a top_k): the maxima of a thread's next `every` chunks. The top_k-th largest of them bounds the row's top_k-th
    // largest logit from below, closely (thousands of groups), at a store per group instead of an atomic per logit.
    const int n_it = (c1 - c0 + B - 1) / B;
    s.every = max(1, (n_it * B + kCGroups - 1) / kCGroups);
    s.list_n[0] = 0u; s.list_n[1] = 0u;
    s.o_tau = -INFINITY; s.o_token = -1; s.o_weight = 0ull; s.few = (call & kCallFew) != 0u;
    s.o_status = (s.want_stats ? LM_STATUS_GENERIC_PATH : 0u) | (s.few ? LM_STATUS_SLICED_PATH : 0u);   // (statistics: what such calls have always reported)
  }
  {                                                                         // the slice starts its way into L2 (a thread's loads have two chunks in flight)
    const int lo_b = max(0, 8 * c0 - off) * (F32 ? 4 : 2), hi_b = min(V, 8 * c1 - off) * (F32 ? 4 : 2);
    for (int l = lo_b + tid * 128; l < hi_b; l += B * 128) prefetch_l2_line(rowp + l);
  }
  if (pen_on) {
    uint32_t* w = reinterpret_cast<uint32_t*>(pen);
    for (int i = tid; i < (per + 3) / 4; i += B) w[i] = 0u;
    __syncthreads();
    const int32_t* h = P.history + static_cast<int64_t>(row) * P.hist_stride;
    for (int i = tid; i < P.hist_len; i += B) {
      const int id = __ldg(h + i);
      const int j = id + off - 8 * c0;
      if (id >= 0 && id < V && j >= 0 && j < 8 * (c1 - c0)) atomicOr(&w[j >> 5], 1u << (j & 31));
    }
  }
  __syncthreads();

  bool ok = V > 0 && T >= 0.0f;
  if (ok) { phase_load<F32, CACHED, B>(s); ok = !s.fallback; }
  else if (C > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  double kept_mass = 1.0;
  if (ok && T == 0.0f) {                                                    // greedy
    if (tid == 0) s.o_token = s.arg;
    if (P.out_probs) phase_probs<F32, CACHED>(s, P, s.arg, 1.0);
  } else if (ok) {
    const bool listy = s.has_k && s.top_k <= kCListK && !(P.flags & LM_FLAG_EXACT_ONLY);
    bool done = false;
    if (listy) {
      bool written;
      done = phase_top_k<F32, CACHED, B>(s, P, &written);
      if (written) {
        if (C > 1) cluster_sync(C);                                         // no block leaves while another may still read or write its memory
        return;
      }
    }
    if (!done) ok = phase_search<F32, CACHED, B>(s, listy);
    if (ok && s.want_stats) {
      kept_mass = done ? s.kept_mass : phase_mass64<F32, CACHED>(s, s.o_tau, s.x_kept);   // (a list of the top-k set has it already)
      if (P.out_probs) phase_probs<F32, CACHED>(s, P, -1, 1.0 / kept_mass);
    }
  }
  if (!ok) {
    cluster_sync(C);                                                        // rank 0's shared memory is written over: nobody may still push into it
    if (rank == 0) generic_row_fallback(P, s, smem_raw);
    return;
  }
  __syncthreads();
  if (rank == 0 && tid == 0) {
    store_token(P.out_tokens, P.flags, row, s.o_token);
    if (P.out_tau) P.out_tau[row] = s.o_tau;
    if (P.out_stats) { P.out_stats[2 * row] = s.vmax; P.out_stats[2 * row + 1] = static_cast<float>(kept_mass); }
    if (P.out_vmax) P.out_vmax[row] = s.vmax;
    if (P.out_mass) P.out_mass[row] = s.o_weight;
    if (P.out_status) P.out_status[row] = s.o_status;
  }
  if (C > 1) cluster_sync(C);                                               // no block leaves while another may still read or write its memory
}

}  // namespace lm

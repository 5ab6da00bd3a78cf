// The top-k candidate kernel: rows with 1 <= top_k <= kTopkMaxK in ONE pass over the row, no histogram, small blocks.
//
// With top-k on, the kept set lies inside the row's top-k logits. So the pass only has to (a) collect the few logits at or
// above a cutoff (estimated per row from 8192 of its logits: about 1 % of the row ends up above it), and
// (b) accumulate the softmass of the whole row in FP32 (the top-p target needs it). Everything exact then happens on the
// candidates alone: the k-th largest value, FP64 masses, the top-p boundary, integer weights, the draw. The FP32 mass is
// only used to decide on which side of top_p * Z a cumulative mass lies; if that is closer than the FP32 error bound (derived
// where it is applied), the mass is formed again in FP64. If the candidates do not cover the top-k set, or anything else does not
// fit, the row is handed on and the histogram kernel redoes it exactly.
// Two blocks of 512 threads share an SM (~93 KB of shared memory each): the per-row phases after the pass are chains of short
// dependent steps, and only the row in the other block can hide them.
// No counterpart in the reference (its sampler always builds the full histogram, kernels/common/sample.metal:34-162).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"
#include "sample_generic.cuh"
#include "vocab_parallel.cuh"

namespace lm {

constexpr int kTB = 512;                   // threads per block
constexpr int kTopkPerSM = 2;              // blocks per SM (64 registers per thread, ~92 KB of shared memory each)
constexpr int kTW = kTB / 32;
constexpr int kTopkCap = 2048;             // candidates per row (a power of two: the sorts pad to one)
constexpr int kTopkBins = 512;             // BF16 codes above the cutoff that the coarse count covers
constexpr int kTopkMaxK = 1024;            // largest top_k this kernel takes
constexpr int kTopkHist = 2048;            // longest history it takes
constexpr int kTopkMaxVocab = 1 << 18;
constexpr int kSearchProbes = 30;          // counters of the cutoff search per row: three per round, one round for the bracket + eight for the whole code range ...
constexpr int kMaxProbes = kSearchProbes + 7;   // ... and seven for the looks around the cutoff (topk_settle)
constexpr int kBinSortMax = 256;           // most candidates of one code bin whose values are no BF16 values (penalised ones), unless they are in order already (all equal)
constexpr int kFew = 64;                   // this many candidates down to the top-k crossing are finished by one warp
constexpr uint32_t kRefineFrom = 44u;      // sampled logits wanted from which on the cutoff is corrected by as many samples again
constexpr int kSampleChunks = 1024 / kTB;   // chunks per thread in the cutoff sample: 1024 chunks = 8192 logits
static_assert(kSampleChunks == 2, "topk_settle holds a bit for each logit of a thread's two samples");
constexpr int kTopkMinVocab = 32768;

constexpr int kStages = 4;                 // 16-byte asynchronous copies in flight per thread during the pass

struct TopkSmem {
  union {
    struct {
      unsigned long long key[kTopkCap];    // candidates as (monotone value key << 32) | ~index, arrival order; later the draw's index buckets
      unsigned long long sel[kTopkCap];    // those at or above the top-k crossing, in descending value order
    };
    uint4 ring[kStages][kTB];              // during the pass: each thread's own landing slots for its chunks of the row
  };
  union {
    double cum[kTopkCap];                  // FP64 softmass prefix over sel ...
    unsigned long long w[kTopkCap];        // ... then the fixed-point weights of the kept prefix
    uint32_t side_id[kTopkHist];           // before either: the distinct history ids
  };
  uint32_t pen[kTopkMaxVocab / 32];        // bitmap of the row's distinct history ids
  uint32_t hitlist[2048];                  // the chunks that hold a logit >= cutoff
  uint32_t bins[kTopkBins];                // candidates per BF16 code, relative to the cutoff code
  uint32_t off[kTopkBins];                 // candidates in the bins above each bin
  uint64_t scratch[32];
  double warp_d[kTW];
  uint32_t warp_u[kTW];
  uint32_t probe_cnt[kMaxProbes];          // block totals of the cutoff search, one slot per probe
  uint32_t prev_cut[8];                    // the block's last cutoff per size class of the candidate target (0: none yet)
  float warp_f[kTW];
  unsigned long long base;
  uint32_t n_hit, n, n_side, wide, cross_bin, ref_key;
  int hit, token, row;
};

static_assert(kTopkPerSM * (sizeof(TopkSmem) + 1024) <= 233472, "the blocks of the top-k kernel must fit one SM's shared memory");

// What the candidate path knows about the softmass of the whole row when it reaches the exact phases: z_tilde approximates
// sum_i 2^(z_i c + shift'), the exact mass relative to a maximum vmax is z_tilde * 2^(shift - vmax c); z_raw is the part of it
// that was accumulated in FP32 (sequences of acc_terms additions), z_corr what was added and removed term by term (penalties);
// ref is the logit the exponents were taken relative to (a logit of the row at or near its maximum).
// row: its BF16 codes, n_chunks of eight, where the mass can be formed again in FP64 (c.pen marks the penalised positions); nullptr: the logits are gone.
struct RowMass { bool need; double z_tilde, z_raw, z_corr, shift, slope, acc_terms; float ref; const uint16_t* row; int n_chunks; bool penalised; };

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void prefetch_l2_line(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Inclusive FP64 prefix sum over v[0 .. n) in place, n <= kTopkCap, index order; every thread calls (a thread takes consecutive entries).
__device__ __forceinline__ void scan_f64(double* v, int n, double* warp_d) {
  constexpr int kPer = kTopkCap / kTB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double x[kPer], sum = 0.0;
#pragma unroll
  for (int j = 0; j < kPer; j++) { const int i = tid * kPer + j; sum += i < n ? v[i] : 0.0; x[j] = sum; }
  double incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const double t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
  if (lane == 31) warp_d[warp] = incl;
  __syncthreads();
  const double before = warp_sum_f64(lane < warp ? warp_d[lane] : 0.0) + (incl - sum);
#pragma unroll
  for (int j = 0; j < kPer; j++) { const int i = tid * kPer + j; if (i < n) v[i] = before + x[j]; }
  __syncthreads();
}

// Warp-aggregated append: every lane of the warp calls with its count; returns the lane's first slot.
__device__ __forceinline__ uint32_t warp_reserve(uint32_t* counter, uint32_t mine) {
  const int lane = threadIdx.x & 31;
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  uint32_t base = 0u;
  if (lane == 0 && total) base = atomicAdd(counter, total);
  base = __shfl_sync(kFull, base, 0);
  return base + incl - mine;
}

// ... of at most one entry a lane.
__device__ __forceinline__ uint32_t warp_reserve_one(uint32_t* counter, bool mine) {
  const int lane = threadIdx.x & 31;
  const uint32_t votes = __ballot_sync(kFull, mine);
  uint32_t base = 0u;
  if (lane == 0 && votes) base = atomicAdd(counter, __popc(votes));
  return __shfl_sync(kFull, base, 0) + __popc(votes & ((1u << lane) - 1u));
}

// Whether a row is this kernel's at all, from its knobs and address alone (no look at the logits).
__device__ __forceinline__ bool topk_row_eligible(const SampleDev& P, int row) {
  const int V = P.vocab;
  const float T = P.temperature ? P.temperature[row] : P.temperature_s;
  const int top_k = P.top_k ? P.top_k[row] : P.top_k_s;
  const uint16_t* rowp = reinterpret_cast<const uint16_t*>(P.logits) + static_cast<size_t>(row) * static_cast<size_t>(P.row_stride);
  return T > 0.0f && top_k >= 1 && top_k <= kTopkMaxK && (V % kChunk) == 0 && V >= kTopkMinVocab && V <= kTopkMaxVocab &&
         (reinterpret_cast<uintptr_t>(rowp) & 15u) == 0 && !(P.history != nullptr && P.hist_len > kTopkHist);
}

// What the row kernels of a call share in the workspace: the counters begin at zero, the rows that are not the top-k kernel's are listed for the
// histogram kernel. One block: it clears and counts without a memset of its own in front (2 us of every call).
// order: optional, the top-k kernel's own rows in the order in which its blocks take them: those with a large top_k from the front, the others from the back.
constexpr int kPrepThreads = 1024, kCounters = 8, kCounterOther = 4, kCounterLong = 6, kCounterShort = 7;
static __global__ void __launch_bounds__(kPrepThreads) sample_prep_kernel(SampleDev P, int* list, int* counters, int* order) {
  __shared__ int n, n_long, n_short;
  if (threadIdx.x == 0) n = n_long = n_short = 0;
  after_predecessor();
  apply_step_state(P);
  __syncthreads();
  if (threadIdx.x < kCounterOther || threadIdx.x == 5) counters[threadIdx.x] = 0;
  constexpr int kU = 4;                                                     // rows of a thread whose knobs are in flight
  for (int r0 = threadIdx.x; r0 < P.rows; r0 += kU * kPrepThreads) {
    bool other[kU]; int top_k[kU];
#pragma unroll
    for (int j = 0; j < kU; j++) {
      const int row = r0 + j * kPrepThreads;
      other[j] = row < P.rows && !topk_row_eligible(P, row);
      top_k[j] = order != nullptr && row < P.rows && P.top_k ? P.top_k[row] : 0;
    }
#pragma unroll
    for (int j = 0; j < kU; j++) {
      const int row = r0 + j * kPrepThreads;
      if (other[j]) list[atomicAdd(&n, 1)] = row;
      else if (order != nullptr && row < P.rows) order[top_k[j] > kFew ? atomicAdd(&n_long, 1) : P.rows - 1 - atomicAdd(&n_short, 1)] = row;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) { counters[kCounterOther] = n; counters[kCounterLong] = n_long; counters[kCounterShort] = n_short; }
}

// How many logits of the row lie at or above code a (low word) and code b (high word); every thread calls.
static __device__ __noinline__ uint64_t topk_count_row(const uint4* p4, int n_chunks, uint32_t a, uint32_t b, uint64_t* scratch) {
  constexpr int kDeep = 8;                                                  // a thread's loads in flight
  uint32_t na = 0u, nb = 0u;
  for (int c0 = threadIdx.x; c0 < n_chunks; c0 += kDeep * kTB) {
    uint4 q[kDeep];
#pragma unroll
    for (int j = 0; j < kDeep; j++) q[j] = c0 + j * kTB < n_chunks ? __ldg(p4 + c0 + j * kTB) : make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);
#pragma unroll
    for (int j = 0; j < kDeep; j++) { na += __popc(kept_bits8(q[j], a | (a << 16))); nb += __popc(kept_bits8(q[j], b | (b << 16))); }
  }
  return block_sum_u64(static_cast<uint64_t>(na) | (static_cast<uint64_t>(nb) << 32), scratch);
}

// Chunk j of a thread's second sample, between those of the first, and where it lands: the list of the chunks is written behind the pass, and the
// history's ids fill the first half of their array at most.
__device__ __forceinline__ int topk_second_chunk(int tid, int j, int n_chunks) { return tid + (2 * j + 1) * (n_chunks / (2 * kSampleChunks)); }
__device__ __forceinline__ uint4* topk_second_slot(TopkSmem& c, int tid, int j) { return (j ? reinterpret_cast<uint4*>(c.cum + kTopkCap / 2) : reinterpret_cast<uint4*>(c.hitlist)) + tid; }

// The cutoff that the search on one sample has found, looked at again on that sample (q0, q1) and a second one as large (staged: it has been asked
// for). A function of its own: inline it made the rows that never come by up to 10 % slower (350 rows, top_k 100), and the second sample held in
// registers from the start of the row did so too. lam, full: what top_k and kTopkCap logits of the row stand for in one sample. 0: no cutoff will
// do. Every thread calls; the copies in flight have landed behind it.
static __device__ __noinline__ uint32_t topk_settle(const uint4* p4, int n_chunks, int top_k, float lam, float full, uint32_t want, uint32_t cut, bool coarse, bool staged, bool pen_on,
                                                    uint4 q0, uint4 q1, TopkSmem& c) {
  const int tid = threadIdx.x, lane = tid & 31;
  uint4 q[4] = {q0, q1};
  cp_async_wait<0>();
#pragma unroll
  for (int j = 0; j < 2; j++) q[2 + j] = staged ? *topk_second_slot(c, tid, j) : __ldg(p4 + topk_second_chunk(tid, j, n_chunks));
  auto count = [&](int slot, uint32_t code) {
    uint32_t bits = 0u;
#pragma unroll
    for (int j = 0; j < 4; j++) bits |= kept_bits8(q[j], code | (code << 16)) << (4 * j);
    const uint32_t n = warp_sum_u32(__popc(bits));
    if (lane == 0 && n) atomicAdd(&c.probe_cnt[kSearchProbes + slot], n);
  };
  // How far a count lies inside of what the top_k and what the list of candidates stand for, in standard deviations.
  auto inside = [&](uint32_t n) {
    const float low = 2.0f * lam, high = 2.0f * full, x = static_cast<float>(n);
    return fminf((x - low - 2.0f) * rsqrtf(low), (high - x) * rsqrtf(high));
  };
  if (coarse) {
    // Coarse logits: the next code up has fewer than wanted, this one more than the usual slack. Either may be the right side of the step: the
    // upper one where it surely has top_k logits, this one where they surely fit the list, else the row is counted. (256 rows of integers N(0, 2^2), us
    // with one step of the cutoff on the samples alone, which hands half of them on / so: 151,936 logits, top_k 450 411 / 144, 1000 493 / 152; 262,144
    // logits, top_k 100 239 / 51, 300 919 / 75. Counting a row takes about 10 us of it.)
    count(0, cut); count(1, cut + 1u);
    __syncthreads();
    if (inside(c.probe_cnt[kSearchProbes + 1]) >= 3.0f) return cut + 1u;
    if (inside(c.probe_cnt[kSearchProbes]) >= 3.0f) return cut;
    const uint64_t both = topk_count_row(p4, n_chunks, cut, cut + 1u, c.scratch);
    if (static_cast<uint32_t>(both) <= static_cast<uint32_t>(kTopkCap)) return cut;
    if (static_cast<uint32_t>(both >> 32) >= static_cast<uint32_t>(top_k)) return cut + 1u;
    return pen_on ? cut : 0u;                                               // (penalties may yet move some below it)
  }
  // A large top_k has little room on either side (1477 candidates for 1000, of 2048): of the cutoff and its neighbours the one that both samples
  // together put nearest to what is wanted, if it is well inside, or furthest inside; four more where that is less far than it should be (of N(0, 2^2) logits
  // with a top_k of 1000 one row in 300 of 151,936, one in 4 of 262,144). One row in 400 with a top_k of 1000 missed with one sample, and made a
  // call of 256 rows 60 us longer; one in 600 of 262,144 does so now. (Five looks at once: 256 rows, top_k 400 42.9 us, 42.2 so.)
  constexpr int kAt[7] = {0, -5, 5, -2, 2, -10, 10};                        // (a code is 1 to 4 % of the candidates)
  float best = -INFINITY, best_in = 0.0f; int by = 0;
  auto look = [&](int first, int last) {
#pragma unroll
    for (int t = 0; t < 7; t++) if (t >= first && t < last) count(t, cut + kAt[t]);
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 7; t++) if (t >= first && t < last) {
      const uint32_t n = c.probe_cnt[kSearchProbes + t];
      const float in = inside(n), fit = in >= 3.0f ? -fabsf(static_cast<float>(n) - 2.0f * static_cast<float>(want)) : in - 1e6f;
      if (fit > best) { best = fit; best_in = in; by = kAt[t]; }
    }
  };
  look(0, 3);
  if (best_in < 2.5f) look(3, 7);                                           // (uniform)
  return max(static_cast<uint32_t>(static_cast<int>(cut) + by), 0x0080u);
}

struct TopkSmem;
static __device__ bool topk_finish(const SampleDev& P, int row, TopkSmem& c, uint32_t cut_code, const RowMass& zm);

// One row. Every thread of the block calls with the same arguments; returns true when the row is finished, false when the
// histogram kernel has to take it (nothing has been written then).
// `next` is the row this block takes afterwards (-1: none): its sample and history are pulled into L2 meanwhile.
static __device__ bool topk_row(const SampleDev& P, int row, int next, TopkSmem& c) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int V = P.vocab;
  const float T = P.temperature ? P.temperature[row] : P.temperature_s;
  const int top_k = P.top_k ? P.top_k[row] : P.top_k_s;
  const float top_p = P.top_p ? P.top_p[row] : P.top_p_s;
  const float min_p = P.min_p ? P.min_p[row] : P.min_p_s;
  const uint16_t* rowp = reinterpret_cast<const uint16_t*>(P.logits) + static_cast<size_t>(row) * static_cast<size_t>(P.row_stride);
  const bool pen_on = P.history != nullptr;
  const int n_chunks = V / kChunk;
  const uint4* p4 = reinterpret_cast<const uint4*>(rowp);
  const bool has_p = top_p > 0.0f && top_p < 1.0f, has_m = min_p > 0.0f;
  const bool in_topk = (P.flags & LM_FLAG_TOPP_IN_TOPK) && has_p;
  const bool need_z = has_p && !in_topk;
  const double T64 = static_cast<double>(T), inv_t = 1.0 / T64;
  const float c2a = static_cast<float>(1.4426950408889634 * inv_t);          // the FP32 softmass only: approximate on purpose

  // the first chunks of the pass do not depend on the cutoff: they start now and land in this thread's slots
  const int n_it = (n_chunks + kTB - 1) / kTB;
#pragma unroll
  for (int it = 0; it < kStages - 1; it++) {
    if (it * kTB + tid < n_chunks) cp_async16(&c.ring[it][tid], p4 + it * kTB + tid);
    cp_async_commit();
  }
  if (next >= 0) {
    const uint4* np4 = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(P.logits) + static_cast<size_t>(next) * static_cast<size_t>(P.row_stride));
    if ((tid & 7) == 0) {                                                   // one prefetch per 128-byte line of the sample runs
#pragma unroll
      for (int j = 0; j < kSampleChunks; j++) prefetch_l2_line(np4 + tid + j * (n_chunks / kSampleChunks));
    }
    if (pen_on && tid * 32 < P.hist_len) prefetch_l2_line(P.history + static_cast<int64_t>(next) * P.hist_stride + tid * 32);
  }
  // ---- the cutoff sample goes out first; the bitmap and the list of the history's distinct ids are built under its latency ---
  // (runs of chunks spread over the row: token ids are not exchangeable in a real vocabulary)
  uint4 qs[kSampleChunks];
#pragma unroll
  for (int j = 0; j < kSampleChunks; j++) qs[j] = __ldg(p4 + tid + j * (n_chunks / kSampleChunks));
  // The sampled logits wanted at or above the cutoff: what the top_k stands for in the sample (lam), and so many more that one row in 10^5 has fewer
  // than top_k candidates (4.3 standard deviations of a Poisson count, and 6 for the small ones), but no more than lie as many of its standard deviations
  // above that as below what the list of candidates holds (the means of square roots: the spread of a count's root is the same everywhere).
  const float per_logit = static_cast<float>(kSampleChunks * kTB * kChunk) / static_cast<float>(V), lam = static_cast<float>(top_k) * per_logit, full = static_cast<float>(kTopkCap) * per_logit;
  const float middle = 0.5f * (sqrtf(lam) + sqrtf(full));
  const uint32_t want = static_cast<uint32_t>(fminf(ceilf(lam + 4.3f * sqrtf(lam) + 6.0f), middle * middle));
  const bool refine = want >= kRefineFrom || (static_cast<float>(want) - lam - 2.0f) < 4.0f * sqrtf(lam);   // ... or less slack than usual
  if (refine) {                                                             // as many samples again, between the others, land where nothing else does before the pass
#pragma unroll
    for (int j = 0; j < kSampleChunks; j++) cp_async16(topk_second_slot(c, tid, j), p4 + topk_second_chunk(tid, j, n_chunks));
    cp_async_commit();
  }
  constexpr int kHistPer = kTopkHist / kTB;
  int hid[kHistPer];                                                        // this thread's share of the history, in flight with the sample
#pragma unroll
  for (int j = 0; j < kHistPer; j++) {
    const int i = tid + j * kTB;
    hid[j] = (pen_on && i < P.hist_len) ? __ldg(P.history + static_cast<int64_t>(row) * P.hist_stride + i) : -1;
  }
  for (int i = tid; i < kTopkBins; i += kTB) c.bins[i] = 0u;
  if (tid < kMaxProbes) c.probe_cnt[tid] = 0u;
  if (pen_on) {
    uint4* p = reinterpret_cast<uint4*>(c.pen);
    for (int i = tid; i < (V + 127) / 128; i += kTB) p[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid == 0) { c.n_hit = 0u; c.n = 0u; c.n_side = 0u; c.wide = 0u; c.ref_key = 0u; c.hit = kTopkCap; c.token = -1; c.cross_bin = 0u; }
  __syncthreads();
  // the thread that sets an id's bit owns the id and lists it
#pragma unroll
  for (int j = 0; j < kHistPer; j++) {
    const int id = hid[j];
    bool fresh = false;
    if (id >= 0 && id < V) {
      const uint32_t bit = 1u << (id & 31);
      fresh = (atomicOr(&c.pen[id >> 5], bit) & bit) == 0u;
    }
    const uint32_t slot = warp_reserve_one(&c.n_side, fresh);
    if (fresh) c.side_id[slot] = static_cast<uint32_t>(id);
  }
  // ---- the cutoff: the largest positive BF16 code with at least `want` of the 8192 sampled logits at or above it ---------
  // A bisection over the codes, one barrier per probe; it starts from a bracket around the cutoff of the block's last
  // row of the same size class, which usually holds (rows of one batch come from one model), and costs ~7 probes then.
  uint32_t cut_code;
  {
    const int cls = min(31 - __clz(want), 7);
    int probe = 0;
    // sampled logits at or above each of three codes, with one barrier; every thread calls
    auto count_in = [&](const uint4 (&q)[kSampleChunks], uint32_t code) {
      uint32_t bits = 0u;                                                   // a bit per logit, gathered first: a count of bits takes four times as long as a logical operation
#pragma unroll
      for (int j = 0; j < kSampleChunks; j++) bits |= kept_bits8(q[j], code | (code << 16)) << (4 * j);
      return static_cast<uint32_t>(__popc(bits));
    };
    auto count3 = [&](uint32_t a, uint32_t b, uint32_t d, uint32_t out[3]) {
      const uint32_t codes[3] = {a, b, d};
#pragma unroll
      for (int t = 0; t < 3; t++) {
        const uint32_t n = warp_sum_u32(count_in(qs, codes[t]));
        if (lane == 0 && n) atomicAdd(&c.probe_cnt[probe + t], n);
      }
      __syncthreads();
#pragma unroll
      for (int t = 0; t < 3; t++) out[t] = c.probe_cnt[probe + t];
      probe += 3;
    };
    // the largest sampled logit: the reference point of the FP32 softmass (any value near the row maximum will do); it
    // travels with the first barrier
    __nv_bfloat162 mx = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&qs[0].x), *reinterpret_cast<const __nv_bfloat162*>(&qs[0].y));
    mx = __hmax2(mx, __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&qs[0].z), *reinterpret_cast<const __nv_bfloat162*>(&qs[0].w)));
#pragma unroll
    for (int j = 1; j < kSampleChunks; j++) {
      mx = __hmax2(mx, __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&qs[j].x), *reinterpret_cast<const __nv_bfloat162*>(&qs[j].y)));
      mx = __hmax2(mx, __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&qs[j].z), *reinterpret_cast<const __nv_bfloat162*>(&qs[j].w)));
    }
    const float mine_max = fmaxf(__low2float(mx), __high2float(mx));
    const uint32_t max_key = warp_max_u32(fkey(mine_max));
    if (lane == 0) atomicMax(&c.ref_key, max_key);
    // A few candidates more than wanted cost less than another round: a cut is good enough at twice the count wanted while that is small, at half
    // as much again beyond; a large top_k's is corrected below. Never more than stand for 1500 candidates in the row: the list holds 2048,
    // and at the largest vocabularies a sampled logit stands for 32 (512 rows of 262,144, top_k 1000: 60 rows handed on without that bound, 8 with it).
    const uint32_t most = static_cast<uint32_t>(1500ll * kSampleChunks * kTB * kChunk / V);
    const uint32_t enough = refine ? want + want / 4u : max(want, min(want < 24u ? 2u * want : want + want / 2u, most));
    uint32_t n_lo = 0xFFFFFFFFu;                                            // count(sample >= lo), once it is known
    uint32_t lo = 0x0000u, hi = 0x7F7Fu;                                    // invariant: count(sample >= lo) >= want, or lo is still 0 (handed back below)
    const uint32_t prev = c.prev_cut[cls];
    uint32_t n3[3];
    if (prev >= 0x0080u) {                                                  // both ends of the bracket and its middle in one round
      const uint32_t blo = max(prev, 0x0090u) - 16u, bhi = min(prev + 15u, 0x7F7Eu), mid = (blo + bhi + 1u) >> 1;
      count3(blo, mid, bhi + 1u, n3);
      if (n3[0] < want) hi = blo - 1u;
      else if (n3[2] >= want) { lo = bhi + 1u; n_lo = n3[2]; }
      else if (n3[1] >= want) { lo = mid; hi = bhi; n_lo = n3[1]; }
      else { lo = blo; hi = mid - 1u; n_lo = n3[0]; }
    }
    else {
      // The block's first row of its class: the want-th largest of the threads' own maxima has at least `want` samples at or above it, and seldom
      // many more. One warp finds it (a bisection by four over the three binades below the largest, or over all codes). Without it the search
      // began with every code: 7.9 us of a row's 40 where a block has one row (256 penalised rows), 4.8 so.
      uint16_t* maxima = reinterpret_cast<uint16_t*>(c.off);
      maxima[tid] = mine_max > 0.0f ? static_cast<uint16_t>(__float_as_uint(mine_max) >> 16) : static_cast<uint16_t>(0u);
      __syncthreads();
      const uint32_t top_code = c.ref_key & 0x80000000u ? min((c.ref_key & 0x7FFFFFFFu) >> 16, 0x7F7Fu) : 0u;   // (a NaN or +inf maximum: handed on by the pass)
      if (warp == 0) {
        const uint4 a = reinterpret_cast<const uint4*>(maxima)[2 * lane], b = reinterpret_cast<const uint4*>(maxima)[2 * lane + 1];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        auto at_or_above = [&](uint32_t code) {                            // per lane; two packed counts
          const uint32_t m2 = code | (code << 16);
          const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&m2);
          uint32_t n = 0u;
#pragma unroll
          for (int k = 0; k < 8; k++) n += __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[k]), t2) & 0x00010001u;
          return (n & 0xFFFFu) + (n >> 16);
        };
        uint32_t first = top_code > 0x0080u + 383u ? top_code - 383u : 0x0080u, last = max(top_code, 0x0080u);
        if (warp_sum_u32(at_or_above(first)) < want) { last = first; first = 0x0080u; }
#pragma unroll 1
        while (first < last) {
          const uint32_t span = last - first, q1 = first + (span + 3u) / 4u, q2 = first + (2u * span + 3u) / 4u, q3 = first + (3u * span + 3u) / 4u;
          const uint32_t n = warp_sum_u32(at_or_above(q1) | (at_or_above(q2) << 10) | (at_or_above(q3) << 20));   // (512 at most each)
          if ((n >> 20) >= want) first = q3;
          else if (((n >> 10) & 1023u) >= want) { first = q2; last = q3 - 1u; }
          else if ((n & 1023u) >= want) { first = q1; last = q2 - 1u; }
          else last = q1 - 1u;
        }
        if (lane == 0) c.cross_bin = first;
      }
      __syncthreads();
      lo = c.cross_bin; hi = max(top_code, lo);
      const uint32_t q2 = min(lo + 6u, hi), q3 = min(lo + 18u, hi);
      count3(lo, q2, q3, n3);
      if (n3[2] >= want) { lo = q3; n_lo = n3[2]; }
      else if (n3[1] >= want) { lo = q2; hi = q3 - 1u; n_lo = n3[1]; }
      else if (n3[0] >= want) { hi = q2 - 1u; n_lo = n3[0]; }
      else lo = hi = 0u;                                                    // fewer positive samples than wanted
    }
    while (lo < hi && n_lo > enough && probe + 3 <= kSearchProbes) {          // three cuts per round: the range shrinks fourfold
      const uint32_t span = hi - lo;
      const uint32_t q1 = lo + (span + 3u) / 4u, q2 = lo + (2u * span + 3u) / 4u, q3 = lo + (3u * span + 3u) / 4u;   // lo < q1 <= q2 <= q3 <= hi
      count3(q1, q2, q3, n3);
      if (n3[2] >= want) { lo = q3; n_lo = n3[2]; }
      else if (n3[1] >= want) { lo = q2; hi = q3 - 1u; n_lo = n3[1]; }
      else if (n3[0] >= want) { lo = q1; hi = q2 - 1u; n_lo = n3[0]; }
      else hi = q1 - 1u;
    }
    cut_code = lo;
    if (cut_code < 0x0080u || (lo < hi && n_lo > enough)) { cp_async_wait<0>(); return false; }   // fewer positive logits than candidates wanted: not this kernel's row
                                                                            // (the copies in flight must land before the slots are used again)
    const bool coarse = n_lo > enough;                                      // the next code up has too few, this one more than the usual slack
    if (coarse || refine) {
      cut_code = topk_settle(p4, n_chunks, top_k, lam, full, want, cut_code, coarse, refine, pen_on, qs[0], qs[1], c);
      if (cut_code == 0u) return false;
    }
    if (tid == 0) c.prev_cut[cls] = cut_code;
  }
  const float cut_val = __uint_as_float(cut_code << 16);

  // ---- the one pass: note the chunks that hold a logit >= cutoff; FP32 softmass relative to the sampled maximum ----------
  const float M = need_z ? fkey_inv(c.ref_key) : 0.0f;
  const float nb = -M * c2a;
  // A chunk's terms are added up before they join the thread's sum: as many additions as one after the other, but a term goes through a fourth of them, and
  // their rounding is most of the band inside which a boundary takes the FP64 mass, 35 us more for its row (151,936 logits: the band is 5.5e-6 of the mass so, 1.4e-5 one
  // after the other; of 60 calls of 256 penalised rows ten had such a row, now two, and the calls' mean went from 72.1 to 67.5 us). Finer sums -- chunks in fours, or the steps in turn on two or four accumulators -- cost the pass 0.5 to 2 % (4096 penalised rows, us: 634 so, 638, 640 and 647).
  float2 sacc = make_float2(0.0f, 0.0f);
  uint32_t nan_seen = 0u;
  // A bit per step: this thread's chunk held a logit >= cutoff. The list of those chunks is written behind the pass, one reservation per
  // warp: nearly every step some lane has one, and a reservation per step would be a quarter of the pass's instructions (4096 penalised rows, three
  // in four with a top_k: 857 us with it, 797 without; 64 rows of 262,144, top_k 50: 51 and 45).
  static_assert(kTopkMaxVocab / kChunk <= 64 * kTB, "a bit for every step");
  unsigned long long hits = 0ull;
  {
    const uint32_t cut2 = cut_code | (cut_code << 16);
    const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&cut2);
    const uint4 pad = make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);   // -inf
#pragma unroll 4
    for (int it = 0; it < n_it; it++) {
      {
        const int ahead = it + kStages - 1, ca = ahead * kTB + tid;         // refill the slot read one step ago
        if (ca < n_chunks) cp_async16(&c.ring[ahead % kStages][tid], p4 + ca);
        cp_async_commit();
      }
      cp_async_wait<kStages - 1>();                                         // this step's chunk has landed
      const int cc = it * kTB + tid;
      const uint4 q = cc < n_chunks ? c.ring[it % kStages][tid] : pad;
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      const uint32_t m0 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[0]), t2), m1 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[1]), t2);
      const uint32_t m2 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[2]), t2), m3 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[3]), t2);
      hits = (hits << 1) | ((m0 | m1 | m2 | m3) != 0u ? 1ull : 0ull);       // (the padding is below every cutoff)
      if (need_z) {                                                         // (the padding is -inf: weight 0; a NaN or +inf logit poisons the sum)
        float2 t;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float2 x = __ffma2_rn(make_float2(bf16_lo(w[k]), bf16_hi(w[k])), make_float2(c2a, c2a), make_float2(nb, nb));
          const float2 e = make_float2(ex2_approx(x.x), ex2_approx(x.y));
          t = k ? __fadd2_rn(t, e) : e;
        }
        sacc = __fadd2_rn(sacc, t);
      } else {                                                              // no mass wanted: the NaN check on its own
        const __nv_bfloat162 a = __hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&w[0]), *reinterpret_cast<const __nv_bfloat162*>(&w[1]));
        const __nv_bfloat162 b = __hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&w[2]), *reinterpret_cast<const __nv_bfloat162*>(&w[3]));
        const __nv_bfloat162 ab = __hmax2_nan(a, b);
        nan_seen |= ~__heq2_mask(ab, ab);                                   // a NaN anywhere in the chunk survives the maxima
      }
    }
    cp_async_wait<0>();
  }
  {
    uint32_t slot = warp_reserve(&c.n_hit, static_cast<uint32_t>(__popcll(hits)));
    for (unsigned long long m = hits; m; m &= m - 1ull, slot++)
      if (slot < 2048u) c.hitlist[slot] = static_cast<uint32_t>((n_it - __ffsll(static_cast<long long>(m))) * kTB + tid);
  }
  // a NaN or +inf logit (or a logit far above the sampled maximum) has made this thread's sum NaN or infinite: the exact path
  // takes such rows and reports them
  double zsum = 0.0, zadd = 0.0, zsub = 0.0;                                // the pass's mass; what the penalised logits add; what their raw values had added
  if (need_z) {
    const float total = sacc.x + sacc.y;
    if (!(total < INFINITY)) nan_seen = 1u;
    zsum = static_cast<double>(total);
  }
  if (__syncthreads_or(nan_seen != 0u)) return false;                       // rows with a NaN go to the exact path, which reports them
  const uint32_t n_hit = c.n_hit;                                           // (complete: every warp is past the pass)
  if (n_hit > 2048u) return false;

  // the raw logits of the penalised positions are fetched now, after the pass (the row has just gone through L2), and used
  // behind the expansion below: both sets of loads are in flight together
  constexpr int kGather = kTopkHist / kTB;
  uint32_t ids[kGather]; uint16_t raws[kGather];
  if (pen_on) {
#pragma unroll
    for (int j = 0; j < kGather; j++) {
      const uint32_t i = j * kTB + tid;
      ids[j] = i < c.n_side ? c.side_id[i] : 0u;
      raws[j] = __ldg(rowp + ids[j]);
    }
  }
  // ---- the noted chunks, expanded: their logits come back from L2; penalised positions are skipped (the hash set knows them)
  constexpr int kExpand = 1024 / kTB;                                       // chunk reloads in flight per thread
  for (uint32_t e0 = 0; e0 < n_hit; e0 += kTB * kExpand) {                  // uniform trip count
    uint32_t ents[kExpand]; uint4 qq[kExpand];
#pragma unroll
    for (int j = 0; j < kExpand; j++) {
      const uint32_t e = e0 + j * kTB + tid;
      ents[j] = (e < n_hit) ? c.hitlist[e] : 0u;
      qq[j] = (e < n_hit) ? __ldg(p4 + ents[j]) : make_uint4(0u, 0u, 0u, 0u);   // (zeros: below every cutoff)
    }
#pragma unroll
    for (int j = 0; j < kExpand; j++) {
      if (e0 + j * kTB + warp * 32 >= n_hit) break;                         // warp-uniform
      const uint32_t cc = ents[j], mask = kept_mask8(qq[j], cut_code | (cut_code << 16));
      const uint32_t keep = pen_on ? mask & ~((c.pen[cc >> 2] >> ((cc & 3u) * 8u)) & 0xFFu) : mask;   // penalised positions come from the list
      uint32_t slot = warp_reserve(&c.n, __popc(keep));
      for (uint32_t m = keep; m; m &= m - 1u) {                             // usually one bit
        const uint32_t b = __ffs(m) - 1u;
        const uint32_t word = b < 4u ? (b < 2u ? qq[j].x : qq[j].y) : (b < 6u ? qq[j].z : qq[j].w);
        const float value = (b & 1u) ? bf16_hi(word) : bf16_lo(word);
        if (slot < kTopkCap) c.key[slot] = (static_cast<unsigned long long>(fkey(value)) << 32) | (0xFFFFFFFFu - (cc * kChunk + b));
        slot++;
        const uint32_t rel = (__float_as_uint(value) >> 16) - cut_code;
        if (rel >= kTopkBins) c.wide = 1u; else atomicAdd(&c.bins[rel], 1u);
      }
    }
  }
  // ---- the penalised logits, from the list ---------------------------------------------------------------------------------
  if (pen_on) {
    const uint32_t n_side = c.n_side;
#pragma unroll
    for (int j = 0; j < kGather; j++) {
      const uint32_t i = j * kTB + tid;
      if (j * kTB + warp * 32 >= n_side) break;                             // warp-uniform
      float v = -INFINITY;
      if (i < n_side) {
        const float raw = __uint_as_float(static_cast<uint32_t>(raws[j]) << 16);
        v = penalise(raw, P.rho, P.pi);
        if (need_z) { zadd += static_cast<double>(ex2_approx(__fmaf_rn(v, c2a, nb))); zsub += static_cast<double>(ex2_approx(__fmaf_rn(raw, c2a, nb))); }
      }
      const bool cand = v >= cut_val;
      const uint32_t slot = warp_reserve_one(&c.n, cand);
      if (cand) {
        if (slot < kTopkCap) c.key[slot] = (static_cast<unsigned long long>(fkey(v)) << 32) | (0xFFFFFFFFu - ids[j]);
        const uint32_t rel = (__float_as_uint(v) >> 16) - cut_code;
        if (rel >= kTopkBins) c.wide = 1u; else atomicAdd(&c.bins[rel], 1u);
      }
    }
  }
  double z_raw = 0.0, z_add = 0.0, z_sub = 0.0;                             // block totals, relative to the sampled maximum
  if (need_z) {
    zsum = warp_sum_f64(zsum); zadd = warp_sum_f64(zadd); zsub = warp_sum_f64(zsub);
    double* sd = reinterpret_cast<double*>(c.scratch);
    __syncthreads();
    if (lane == 0) { sd[warp] = zsum; sd[kTW + warp] = zadd; c.warp_d[warp] = zsub; }
    __syncthreads();
    static_assert(kTW == 16, "two of the three sums side by side in a warp");
    double two = sd[lane], third = lane < kTW ? c.warp_d[lane] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) { two += __shfl_xor_sync(kFull, two, o); third += __shfl_xor_sync(kFull, third, o); }
    z_raw = __shfl_sync(kFull, two, 0); z_add = __shfl_sync(kFull, two, 16); z_sub = __shfl_sync(kFull, third, 0);
  }
  const double z_tilde = z_raw - z_sub + z_add;
  if (need_z && !(z_tilde > 0.0)) return false;                             // nothing left after the corrections (cancellation): the exact path
  __syncthreads();
  RowMass zm;
  zm.need = need_z; zm.z_tilde = z_tilde; zm.z_raw = z_raw; zm.z_corr = z_sub + z_add; zm.shift = -static_cast<double>(nb); zm.slope = static_cast<double>(c2a);
  zm.ref = M; zm.acc_terms = n_it + 5.0; zm.row = rowp; zm.n_chunks = n_chunks; zm.penalised = pen_on;
  return topk_finish(P, row, c, cut_code, zm);
}

// The row's softmass in FP64, for the rare row (one in some 4000 of the benchmark's) whose top-p boundary the FP32 mass cannot decide. ~15 FP64 operations per
// logit from L2: less than the histogram kernel would take for the whole row, and behind no other launch. The candidates' keys are dead.
static __device__ double topk_exact_mass(const SampleDev& P, TopkSmem& c, const RowMass& zm, float vmax, double inv_t) {
  double* tab = reinterpret_cast<double*>(c.key);
  const int tid = threadIdx.x;
  __syncthreads();
  if (tid < 64) tab[tid] = exp2(static_cast<double>(tid) * 0.015625);
  __syncthreads();
  const uint4* p4 = reinterpret_cast<const uint4*>(zm.row);
  const double vmax64 = static_cast<double>(vmax);
  double m = 0.0;
  uint4 ahead = tid < zm.n_chunks ? __ldg(p4 + tid) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int cc = tid; cc < zm.n_chunks; cc += kTB) {
    const uint4 q = ahead;
    if (cc + kTB < zm.n_chunks) ahead = __ldg(p4 + cc + kTB);
    const uint32_t bits = zm.penalised ? (c.pen[cc >> 2] >> ((cc & 3) * 8)) & 0xFFu : 0u, w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < kChunk; e++) {
      float z = (e & 1) ? bf16_hi(w[e >> 1]) : bf16_lo(w[e >> 1]);
      if ((bits >> e) & 1u) z = penalise(z, P.rho, P.pi);
      m += exp64((static_cast<double>(z) - vmax64) * inv_t, tab);
    }
  }
  return block_sum_f64(m, c.scratch);
}

// The FP32 mass of the whole row, moved to the exact maximum, and how far it can be from the exact one (the bound with a quarter added).
__device__ __forceinline__ double topk_row_total(const RowMass& zm, float vmax, double inv_t, double* err) {
  // z_tilde approximates sum_i 2^(z_i c2a + nb); nb's own rounding is a common factor and is taken out exactly here (zm.shift is the true -nb,
  // not M c2a).
  const double c64 = 1.4426950408889634 * inv_t;
  // With the slope that the terms were formed with: log2(e) / T in FP64 instead would leave the factor 2^(vmax (c2a - c)), which no
  // bound below holds (a maximum of 105 at T 0.3: 2e-5).
  const double total = zm.z_tilde * exp2(zm.shift - static_cast<double>(vmax) * zm.slope);
  // What separates it from sum_i 2^((z_i - vmax) c), relative, first order, worst case (u = 2^-24, the FP32 unit roundoff):
  //   - c2a = fl32(c): every term is off by a factor 2^(x_i delta), |delta| <= u, x_i = (z_i - M) c; weighted by the terms that is
  //     ln2 u E_w|x| <= u (ln V + 2 ln2 D): E_w[-x ln2] = H - ln Z <= ln V (H the entropy of the softmax, Z >= 1 relative to the
  //     row maximum, V <= 2^18: ln V <= 12.5), and the terms above the sampled maximum have 0 < x <= D = (vmax - M) c;
  //   - the FMA rounds its result: half an ulp of |x| < 32 is at most 2^-20, a factor 2^(2^-20) = 1 + 6.6e-7 on the term, and D / 16 times
  //     that for the terms up to D above the sampled maximum; the terms below -32 weigh less than V 2^-32 altogether;
  //   - ex2.approx.ftz.f32: 2 ulp = 4 u;
  //   - each lane adds its terms up in FP32, then the lanes meet in FP64: the additions that a term goes through, times u (zm.acc_terms: the
  //     pass's 3 in a chunk, one a step, the two halves, and one to spare);
  // These are relative to the mass the pass summed (z_raw), which holds the penalised positions at their raw values. The penalised
  // logits then enter as z_raw - z_sub + z_add, every term of z_sub and z_add with the per-term errors above (FMA, ex2, c2a on a
  // single term: 1.6e-6 covers them for |x| < 32); when penalised tokens carried most of the raw mass the band grows with them.
  // A boundary of the cumulative mass inside the band is decided by the FP64 mass.
  const double u = 5.9604644775390625e-8;
  const double D = fmax(0.0, (static_cast<double>(vmax) - static_cast<double>(zm.ref)) * c64);
  const double rel = u * (12.5 + 1.3862943611198906 * D) + 6.6e-7 * fmax(1.0, D * 0.0625) + 4.0 * u + zm.acc_terms * u;
  *err = 1.25 * (rel * zm.z_raw + 1.6e-6 * zm.z_corr) * (total / zm.z_tilde);
  return total;
}

// At most kFew candidates down to the top-k crossing: ordered by rank, then one warp does the rest with shuffles and votes
// (vocab_parallel.cuh) where the block-wide code needs a barrier per step. Every thread calls. (Rows of 151,936 with a top_k of 20, two blocks to an
// SM: 9.3 us of 32.7 by the block, 5.6 so.)
static __device__ bool topk_finish_few(const SampleDev& P, int row, TopkSmem& c, uint32_t cut_code, const RowMass& zm, int n, uint32_t cross, int n_sel) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < kFew) c.off[tid] = 0u;                                          // (the ranks; everyone has read what was there)
  for (int i = tid; i < n; i += kTB) {
    const unsigned long long k = c.key[i];
    const uint32_t rel = (__float_as_uint(fkey_inv(static_cast<uint32_t>(k >> 32))) >> 16) - cut_code;
    if (rel >= cross) c.sel[atomicAdd(&c.n_hit, 1u)] = k;                   // (n_sel of them)
  }
  __syncthreads();
  {
    const int e = tid % kFew;
    if (e < n_sel) {
      const unsigned long long k = c.sel[e];
      uint32_t r = 0u;
      for (int j = tid / kFew; j < n_sel; j += kTB / kFew) r += c.sel[j] > k ? 1u : 0u;
      if (r) atomicAdd(&c.off[e], r);
    }
  }
  __syncthreads();
  if (tid < n_sel) c.w[c.off[tid]] = c.sel[tid];
  __syncthreads();
  const float T = P.temperature ? P.temperature[row] : P.temperature_s, top_p = P.top_p ? P.top_p[row] : P.top_p_s, min_p = P.min_p ? P.min_p[row] : P.min_p_s;
  const int top_k = P.top_k ? P.top_k[row] : P.top_k_s;
  const double inv_t = 1.0 / static_cast<double>(T);
  const bool has_p = top_p > 0.0f && top_p < 1.0f, in_topk = (P.flags & LM_FLAG_TOPP_IN_TOPK) && has_p;
  MergeTail t;
  t.key = c.w; t.vmax = fkey_inv(static_cast<uint32_t>(c.w[0] >> 32)); t.z_total = 0.0;
  double exact = 0.0;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
    if (warp == 0) {
      VpMergeDev M;
      M.flags = P.flags; M.draw = P.draw; M.uniforms = P.uniforms; M.seed = P.seed; M.step = P.step; M.row_offset = P.row_offset;
      M.out_tokens = P.out_tokens; M.out_tau = P.out_tau; M.out_status = P.out_status; M.out_vmax = P.out_vmax; M.out_mass = P.out_mass;
      M.hand_on = 1; M.path_status = pass ? 0u : LM_STATUS_CANDIDATE_PATH; M.mass_band = 0.0;
      t.amb = 0;
      if (pass) t.z_total = exact;
      else if (has_p && !in_topk) { double err; t.z_total = topk_row_total(zm, t.vmax, inv_t, &err); M.mass_band = err / t.z_total; }
      merge_tail_one_warp<2>(M, row, t, n_sel, T, top_k, top_p, min_p, inv_t, 0u);
      if (lane == 0) c.wide = static_cast<uint32_t>(t.amb);
    }
    __syncthreads();
    if (!c.wide) break;
    if (zm.row == nullptr) return false;                                    // too close to call, and nothing finer to look at here
    exact = topk_exact_mass(P, c, zm, t.vmax, inv_t);                       // ... in FP64
  }
  return true;
}

// The exact phases of the candidate path, on what the pass (or a producer of logits tiles, sample_tiles.cuh) has left in shared
// memory: c.key[0 .. c.n) = every logit of the row at or above the cutoff code as (monotone value key << 32) | ~index, c.bins[b] =
// how many of them have BF16 code cut_code + b, c.wide set if one lies beyond the bins. `zm` is what is known about the mass of
// the WHOLE row. Every thread of the block calls with the same arguments; returns true when the row is finished (token, tau
// and status written), false when the exact path has to take it (nothing has been written then).
static __device__ bool topk_finish(const SampleDev& P, int row, TopkSmem& c, uint32_t cut_code, const RowMass& zm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float T = P.temperature ? P.temperature[row] : P.temperature_s;
  const int top_k = P.top_k ? P.top_k[row] : P.top_k_s;
  const float top_p = P.top_p ? P.top_p[row] : P.top_p_s;
  const float min_p = P.min_p ? P.min_p[row] : P.min_p_s;
  const bool has_p = top_p > 0.0f && top_p < 1.0f, has_m = min_p > 0.0f;
  const bool in_topk = (P.flags & LM_FLAG_TOPP_IN_TOPK) && has_p;
  const double T64 = static_cast<double>(T), inv_t = 1.0 / T64;
  const int n = static_cast<int>(c.n);
  if (n > kTopkCap || n < top_k || c.wide) return false;

  // ---- the candidates at or above the top-k crossing, in descending value order: a counting sort by code bin ---------------
  // (the bins are the BF16 codes relative to the cutoff; the crossing is the highest bin b with at least top_k
  // candidates in the bins >= b; inside a bin only penalised values can differ, and one thread puts its bin in order)
  {
    constexpr int kPer = kTopkBins / kTB;                                    // bins per thread, walked from the top
    uint32_t run = 0u, cb[kPer], mine = 0u;
#pragma unroll
    for (int j = 0; j < kPer; j++) { cb[j] = c.bins[kTopkBins - 1 - (kPer * tid + j)]; mine += cb[j]; }
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
    if (lane == 31) c.warp_u[warp] = incl;
    if (tid == 0) c.n_hit = 0u;
    __syncthreads();
    run = warp_sum_u32(lane < warp ? c.warp_u[lane] : 0u);
    uint32_t acc = run + incl - mine;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      c.off[kTopkBins - 1 - (kPer * tid + j)] = acc;
      c.hitlist[kTopkBins - 1 - (kPer * tid + j)] = 0u;                      // (dead since the candidates were expanded: see `front` below)
      if (acc < static_cast<uint32_t>(top_k) && acc + cb[j] >= static_cast<uint32_t>(top_k)) c.cross_bin = static_cast<uint32_t>(kTopkBins - 1 - (kPer * tid + j));
      acc += cb[j];
    }
    __syncthreads();
  }
  const uint32_t cross = c.cross_bin;
  const int n_sel = static_cast<int>(c.off[cross] + c.bins[cross]);
  __syncthreads();                                                          // the counts are consumed below
  if (n_sel <= kFew) return topk_finish_few(P, row, c, cut_code, zm, n, cross, n_sel);
  // In a bin, the values that are no BF16 values (penalised logits) lie above those that are, which are all equal: they fill their bin from its
  // front, the others from its end, and only they have to be put in order.
  uint32_t* front = c.hitlist;
  for (int i = tid; i < n; i += kTB) {
    const unsigned long long k = c.key[i];
    const uint32_t bits = __float_as_uint(fkey_inv(static_cast<uint32_t>(k >> 32))), rel = (bits >> 16) - cut_code;
    if (rel >= cross) c.sel[c.off[rel] + ((bits & 0xFFFFu) ? atomicAdd(&front[rel], 1u) : atomicSub(&c.bins[rel], 1u) - 1u)] = k;
  }
  __syncthreads();
  for (uint32_t b = cross + tid; b < kTopkBins; b += kTB) {
    const uint32_t lo = c.off[b], hi = lo + front[b];
    uint32_t from = lo + 1u;                                                // those in order already (all, if they are equal) stay
    while (from < hi && (c.sel[from - 1u] >> 32) >= (c.sel[from] >> 32)) from++;
    if (from < hi && hi - lo > static_cast<uint32_t>(kBinSortMax)) { c.wide = 1u; continue; }
    for (uint32_t i = from; i < hi; i++) {                                  // insertion sort on the value part
      const unsigned long long k = c.sel[i];
      uint32_t j = i;
      while (j > lo && (c.sel[j - 1u] >> 32) < (k >> 32)) { c.sel[j] = c.sel[j - 1u]; j--; }
      c.sel[j] = k;
    }
  }
  __syncthreads();
  if (c.wide) return false;                                                 // a large bin of unequal (penalised) values: the exact path takes the row
  auto value_at = [&](int i) { return fkey_inv(static_cast<uint32_t>(c.sel[i] >> 32)); };
  // how many of the ordered candidates lie at or above v (complete behind the next barrier; `count` held 0 before the last one)
  auto count_prefix = [&](float v, uint32_t* count) {
    for (int i = tid; i < n_sel; i += kTB) if (value_at(i) >= v && (i == n_sel - 1 || value_at(i + 1) < v)) *count = static_cast<uint32_t>(i + 1);
  };

  // ---- exact thresholds on the sorted candidates ------------------------------------------------------------------------
  const float vmax = fkey_inv(static_cast<uint32_t>(c.sel[0] >> 32));
  const float tau_k = fkey_inv(static_cast<uint32_t>(c.sel[top_k - 1] >> 32));
  double tau64 = tau_k;
  uint32_t status = LM_STATUS_CANDIDATE_PATH;
  if (has_p) {
    for (int i = tid; i < n_sel; i += kTB) c.cum[i] = softmass(fkey_inv(static_cast<uint32_t>(c.sel[i] >> 32)), vmax, inv_t);
    __syncthreads();
    count_prefix(tau_k, &c.n_hit);
    double total = 0.0, err = 0.0;
    if (!in_topk) total = topk_row_total(zm, vmax, inv_t, &err);
    scan_f64(c.cum, n_sel, c.warp_d);                                       // (two barriers)
    const int n_topk = static_cast<int>(c.n_hit);
    if (in_topk) total = c.cum[n_topk - 1];
    double target;
    bool edge = false;
#pragma unroll 1
    for (bool exact = false;; exact = true) {
      target = static_cast<double>(top_p) * total;
      bool amb = false;
      for (int i = tid; i < n_sel; i += kTB) {
        const bool run_end = (i == n_sel - 1) || ((c.sel[i + 1] >> 32) != (c.sel[i] >> 32));
        if (!run_end) continue;
        const double cm = c.cum[i];
        if (cm >= target) atomicMin(&c.hit, i);
        if (!exact && i < n_topk - 1 && fabs(cm - target) <= err && fkey_inv(static_cast<uint32_t>(c.sel[i] >> 32)) > tau_k) amb = true;
        if (exact && fabs(cm - target) <= 1e-12 * total) edge = true;
      }
      if (!__syncthreads_or(amb)) break;
      if (zm.row == nullptr || in_topk) return false;                       // too close to call, and nothing finer to look at here
      total = topk_exact_mass(P, c, zm, vmax, inv_t);                       // ... in FP64
      status = 0u;
      if (tid == 0) c.hit = kTopkCap;
      __syncthreads();
    }
    if (__syncthreads_or(edge)) status |= LM_STATUS_TOPP_EDGE;
    if (c.hit < kTopkCap) {
      const float tau_p = fkey_inv(static_cast<uint32_t>(c.sel[c.hit] >> 32));
      if (static_cast<double>(tau_p) > tau64) tau64 = tau_p;
      if (fabs(c.cum[c.hit] - target) <= 1e-12 * total) status |= LM_STATUS_TOPP_EDGE;
    }
  }
  if (has_m) {
    const double tau_m = static_cast<double>(vmax) + T64 * log(static_cast<double>(min_p));
    if (tau_m > tau64) tau64 = tau_m;
  }
  const float tau = __double2float_rn(tau64);
  if (tid == 0) c.n_side = 0u;
  __syncthreads();
  count_prefix(tau, &c.n_side);
  __syncthreads();
  const int n_kept = static_cast<int>(c.n_side);                            // the kept set is the first n_kept sorted candidates

  // ---- the draw ----------------------------------------------------------------------------------------------------------
  int token = -1;
  uint64_t kept_weight = 0ull;                                             // the kept set's fixed-point mass (for out_mass)
  if (P.draw == LM_DRAW_INVERSE_CDF) {
    // The kept candidates are in descending value order, which is the draw's order up to the order inside a run of equal values
    // (equal values have equal weights): an inclusive prefix sum of the weights finds the candidate where the target is crossed,
    // hence the value; the token is the floor((target - before) / w)-th smallest index of that value's run.
    const float c2 = exp2_scale(T);
    constexpr int kPer = kTopkCap / kTB;                                    // consecutive candidates per thread
    uint64_t wv[kPer], sum = 0ull;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const int i = tid * kPer + j;
      wv[j] = i < n_kept ? weight_q40(fkey_inv(static_cast<uint32_t>(c.sel[i] >> 32)), vmax, c2) : 0ull;
      sum += wv[j];
    }
    uint64_t total = 0ull;
    uint64_t run = block_exclusive_scan_u64(sum, c.scratch, &total);
    kept_weight = total;
    if (tid == 0) { c.hit = kTopkCap; c.cross_bin = 0u; c.n_hit = static_cast<uint32_t>(n_kept); }
    __syncthreads();
    if (total > 0ull) {
      const uint64_t target = cdf_target(P.uniforms ? P.uniforms[row] : 0.0f, total);
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const int i = tid * kPer + j;
        run += wv[j];
        if (i < n_kept) c.w[i] = run;                                       // inclusive
        if (wv[j] && run > target && run - wv[j] <= target) c.hit = i;      // exactly one candidate
      }
      __syncthreads();
      const int at = c.hit;
      const uint32_t vkey = static_cast<uint32_t>(c.sel[at] >> 32);
      // the run of this value: [first, last)
      for (int i = tid; i < n_kept; i += kTB) {
        if (static_cast<uint32_t>(c.sel[i] >> 32) != vkey) continue;
        if (i == 0 || static_cast<uint32_t>(c.sel[i - 1] >> 32) != vkey) c.cross_bin = static_cast<uint32_t>(i);
        if (i == n_kept - 1 || static_cast<uint32_t>(c.sel[i + 1] >> 32) != vkey) c.n_hit = static_cast<uint32_t>(i + 1);
      }
      __syncthreads();
      const int first = static_cast<int>(c.cross_bin), last = static_cast<int>(c.n_hit);
      const uint64_t before = first > 0 ? c.w[first - 1] : 0ull;
      const uint64_t each = c.w[first] - before;
      const uint32_t want = static_cast<uint32_t>((target - before) / each);   // < last - first: the crossing lies inside the run
      for (int i = first + tid; i < last; i += kTB) {
        const uint32_t idx_i = 0xFFFFFFFFu - static_cast<uint32_t>(c.sel[i]);
        uint32_t smaller = 0u;
        for (int t = first; t < last; t++) smaller += (0xFFFFFFFFu - static_cast<uint32_t>(c.sel[t])) < idx_i ? 1u : 0u;
        if (smaller == want) c.token = static_cast<int>(idx_i);
      }
    }
    __syncthreads();
    token = c.token;
  } else {
    const float inv_t32 = __double2float_rn(1.0 / T64);
    const uint32_t t_id = static_cast<uint32_t>(P.row_offset + row);
    uint64_t b1 = 0ull; float second = -INFINITY;
    for (int i = tid; i < n_kept; i += kTB) {
      const unsigned long long k = c.sel[i];
      const uint32_t idx = 0xFFFFFFFFu - static_cast<uint32_t>(k);
      const float key = __fadd_rn(__fmul_rn(fkey_inv(static_cast<uint32_t>(k >> 32)), inv_t32), gumbel(P.seed, P.step, t_id, idx));
      const uint64_t pk = pack_best(key, idx);
      if (pk > b1) { if (b1) second = fmaxf(second, best_value(b1)); b1 = pk; } else second = fmaxf(second, key);
    }
    const uint64_t win = block_max_u64(b1, c.scratch);
    if (win) {
      const float rival = (b1 == win) ? second : (b1 ? best_value(b1) : -INFINITY);
      if (__syncthreads_or(rival >= best_value(win) - 4e-6f)) status |= LM_STATUS_NEAR_TIE;
      token = static_cast<int>(best_index(win));
    }
    if (P.out_mass) {
      const float c2 = exp2_scale(T);
      uint64_t w = 0ull;
      for (int i = tid; i < n_kept; i += kTB) w += weight_q40(fkey_inv(static_cast<uint32_t>(c.sel[i] >> 32)), vmax, c2);
      kept_weight = block_sum_u64(w, c.scratch);
    }
  }
  if (tid == 0) {
    store_token(P.out_tokens, P.flags, row, token);
    if (P.out_tau) P.out_tau[row] = tau;
    if (P.out_status) P.out_status[row] = status;
    if (P.out_vmax) P.out_vmax[row] = vmax;
    if (P.out_mass) P.out_mass[row] = kept_weight;
  }
  __syncthreads();
  return true;
}

// Rows are handed out through a counter in the workspace (counters[0], zeroed by sample_prep_kernel): a block takes
// the next row, passes over it if it is not this kernel's (sample_prep_kernel has listed it), and else either finishes it or appends it to
// `list` (length in counters[1]) for the histogram kernel. The order of the list varies from run to run; what is computed per row does not.
// The row that is taken as the i-th (sample_prep_kernel); rows: there is none.
static __device__ __noinline__ int topk_row_at(const int* order, const int* counters, int rows, int i) {
  const int n_long = __ldcg(counters + kCounterLong), n_short = __ldcg(counters + kCounterShort);   // (from L2: the preparation is two launches back, without an end between)
  return i < n_long ? __ldcg(order + i) : i < n_long + n_short ? __ldcg(order + rows - 1 - (i - n_long)) : rows;
}

// kOrdered: the rows in the order in which they are taken; else all rows as they come (compiled apart: the look-up cost the others 0.3 %).
template <bool kOrdered>
static __global__ void __launch_bounds__(kTB, kTopkPerSM) sample_topk_kernel(SampleDev P, int* list, int* counters, int first, const int* order) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TopkSmem& c = *reinterpret_cast<TopkSmem*>(smem_raw);
  __shared__ int item[2];                                                   // the row in hand and the one after it
  // A histogram kernel launched behind this one with programmatic stream serialization takes over the SMs as this grid's blocks leave them.
  // first: this is the call's first kernel behind sample_prep_kernel, whose counters it needs; else a histogram kernel has begun before it.
  if (first) after_predecessor(); else asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  apply_step_state(P);
  if (threadIdx.x < 8) c.prev_cut[threadIdx.x] = 0u;
  // With many rows per block a block holds the row after its current one too (it pulls that row into L2 while it works) and
  // claims the one after that at the start of a row, so the counter's round trip hides behind the row. With few rows per block
  // claiming ahead would leave blocks without work while others hold two rows: a block then claims a row when it needs one.
  const bool ahead = P.rows >= 4 * static_cast<int>(gridDim.x);
  // Up to three eighths more rows than blocks, all of them this kernel's: the second half of the blocks, which share the SMs of the first (blocks go to all
  // SMs before any has two), leave after a row each, so that a row of the second round has an SM to itself. Else whichever block is done takes the next
  // row, and the two of an SM are done at about the same time. (One top_k for all, us per call so / else: 310 rows, top_k 50 52.3 / 58.3; 350 rows, 50
  // 58.4 / 61.0, 100 56.8 / 59.6, 350 63.2 / 67.2; 400 rows, 100 58.4 / 61.9, 400 64.7 / 68.3, 1000 69.8 / 70.2; with half as many again the first half is too
  // few: 440 rows, top_k 400 74.2 / 64.9.)
  const bool once = first && P.rows * 8LL <= gridDim.x * 11LL && blockIdx.x >= (gridDim.x + 1u) / 2u;
  auto claim = [&]() {                                                      // (thread 0)
    const int i = atomicAdd(&counters[0], 1);
    return kOrdered ? topk_row_at(order, counters, P.rows, i) : i;
  };
  if (threadIdx.x == 0) {
    item[0] = claim();
    item[1] = (ahead && item[0] < P.rows) ? claim() : P.rows;
  }
  __syncthreads();
  for (;;) {
    const int row = item[0], next = item[1];
    if (row >= P.rows) break;
    int fetched = P.rows;
    if (threadIdx.x == 0 && next < P.rows) fetched = claim();
    if (topk_row_eligible(P, row)) {
      const bool done = topk_row(P, row, next < P.rows ? next : -1, c);
      if (threadIdx.x == 0 && !done) list[atomicAdd(&counters[1], 1)] = row;
    }
    __syncthreads();                                                        // nobody reads item[] any more
    if (threadIdx.x == 0) { item[0] = once ? P.rows : ahead ? next : claim(); item[1] = fetched; }
    __syncthreads();
  }
  // This grid may have been started before the grid launched ahead of it had finished (programmatic stream serialization). The
  // stream takes the end of this grid for the end of both, so no block leaves before the earlier grid is complete.
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace lm

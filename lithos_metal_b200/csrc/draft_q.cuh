// Draft-side sampling: the Gumbel-max draw of draft k from the drafter's logits row plus the row statistics (maximum,
// fixed-point mass, log-sum-exp) that let the verify step evaluate q_k(v) later; optionally a copy of the row.
// Follows draft_q_partial / draft_q_final (kernels/common/sample.metal:212-269): same noise stream (2000 + k), same key
// z * float32(1/T) + g; the mass is kept as the integer sum of this library's fixed-point weights instead of an FP32
// running sum, so q_k(v) does not depend on how the row is split.
//
// A few rows of ~300 KB: latency-bound. One thread-block cluster per row (16 blocks for up to 14 rows on 148 SMs), one launch, no
// workspace: a thread holds its few chunks of the row in registers from the one read on, the blocks meet twice in distributed shared
// memory -- the maximum (the weights are relative to it), then mass, best key and runner-up in block 0, which writes the outputs. The
// two logarithms of a Gumbel key are spent only on logits that can still beat the maximum's own key (GumbelScan).
// (A cooperative launch of the whole GPU with a grid barrier, global atomics and both logarithms for every logit took 20 us for 7 rows of
// 151,936, the round of 7 that it opens 58 us; with the cluster 46 to 48.)
#pragma once
#include "sample_cluster.cuh"
#include "spec_ops.cuh"

namespace lm {

constexpr int kDraftQThreads = 512;
constexpr int kDraftQKeep = 4;                          // chunks of eight logits a thread keeps: 16 blocks hold a row of 262,144; the rest is read again from L2

struct DraftQDev {
  int dtype; int rows; int first_position; int vocab; int64_t row_stride;
  const void* logits; float temperature; uint64_t seed; uint32_t step;
  int32_t* out_tokens; float* out_lse; float* out_vmax; unsigned long long* out_mass; uint32_t* out_status;
  void* out_q_logits; int64_t q_logits_stride;
  const uint32_t* state; int t_max, g;                   // optional StepState: seed and step come from it; a done state ends the launch
};

// f(c, raw chunk) for every chunk of this block's slice: the kept ones from registers.
template <bool F32, class F>
__device__ __forceinline__ void draft_chunks(const ClusterRow& R, const RawChunk<F32> (&kept)[kDraftQKeep], F f) {
  const int c = R.c0 + static_cast<int>(threadIdx.x);
#pragma unroll
  for (int j = 0; j < kDraftQKeep; j++) if (c + j * kDraftQThreads < R.c1) f(c + j * kDraftQThreads, kept[j]);
#pragma unroll 1
  for (int d = c + kDraftQKeep * kDraftQThreads; d < R.c1; d += kDraftQThreads) f(d, load_raw<F32>(R, d));
}

template <bool F32>
static __global__ void __launch_bounds__(kDraftQThreads) draft_q_kernel(const DraftQDev P, int C) {
  constexpr int kWarps = kDraftQThreads / 32;
  __shared__ unsigned long long x_best[kCMaxRanks], x_mass[kCMaxRanks], x_key[kCMaxRanks];
  __shared__ float x_rival[kCMaxRanks];
  __shared__ uint32_t x_nan[kCMaxRanks];
  __shared__ uint64_t part_best[kWarps], part_mass[kWarps], part_key[kWarps];
  __shared__ uint32_t part_rival[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0, row = static_cast<int>(blockIdx.x) / C;
  uint64_t seed = P.seed; uint32_t step = P.step;
  after_predecessor();
  if (P.state) {
    StepStateView st{const_cast<uint32_t*>(P.state), P.t_max, P.g};
    if (st.done()) return;                                                  // every block sees the same state
    seed = st.seed(); step = st.step();
  }
  if (C > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this block runs: its memory may be written to
  constexpr int kSize = F32 ? 4 : 2;
  ClusterRow R;
  R.row = static_cast<const char*>(P.logits) + static_cast<size_t>(row) * static_cast<size_t>(P.row_stride) * kSize;
  R.V = P.vocab; R.pen = nullptr; R.rho = 1.0f; R.pi = 0.0f; R.vals = nullptr; R.nv = 0;
  const int head = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(R.row) & 15u)) & 15u) / kSize;
  R.off = head ? 8 - head : 0;
  const int n_chunks = (P.vocab + R.off + 7) / 8, per = (n_chunks + C - 1) / C;
  R.c0 = min(n_chunks, rank * per); R.c1 = min(n_chunks, R.c0 + per);

  // ---- the one read: the slice's maximum (with an index: its Gumbel key is where the draw starts), NaNs -----------------------------
  RawChunk<F32> kept[kDraftQKeep];
#pragma unroll
  for (int j = 0; j < kDraftQKeep; j++) { const int c = R.c0 + tid + j * kDraftQThreads; if (c < R.c1) kept[j] = load_raw<F32>(R, c); }
  uint64_t mine = 0ull;
  bool nan = false;
  draft_chunks<F32>(R, kept, [&](int c, const RawChunk<F32>& q) {
    float z[8];
    widen_raw<F32>(R, q, c, z);
    float mx = z[0];
#pragma unroll
    for (int e = 1; e < 8; e++) asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(mx), "f"(z[e]));
    if (mx != mx) {
      nan = true;
      mx = -INFINITY;
#pragma unroll 1
      for (int e = 0; e < 8; e++) {                                         // the packed order: a positive NaN above +inf, a negative one below -inf
        const int i = 8 * c + e - R.off;
        if (i < 0 || i >= P.vocab) continue;
        const uint64_t p = pack_best(canon_zero(pick8(z, e)), static_cast<uint32_t>(i));
        mine = p > mine ? p : mine;
      }
    } else if (mine == 0ull || mx > best_value(mine)) {
      int at = -1;
#pragma unroll
      for (int e = 7; e >= 0; e--) { const int i = 8 * c + e - R.off; if (z[e] == mx && i >= 0 && i < P.vocab) at = i; }
      if (at >= 0) { const uint64_t p = pack_best(canon_zero(mx), static_cast<uint32_t>(at)); mine = p > mine ? p : mine; }
    }
  });
  if (P.out_q_logits) {                                                     // the copy, element by element (a warp's stores are one line), from L1 / L2
    const int i0 = max(0, 8 * R.c0 - R.off), i1 = min(P.vocab, 8 * R.c1 - R.off);
    for (int i = i0 + tid; i < i1; i += kDraftQThreads) {
      const int64_t o = static_cast<int64_t>(row) * P.q_logits_stride + i;
      if (F32) static_cast<float*>(P.out_q_logits)[o] = __ldg(reinterpret_cast<const float*>(R.row) + i);
      else static_cast<uint16_t*>(P.out_q_logits)[o] = __ldg(reinterpret_cast<const uint16_t*>(R.row) + i);
    }
  }
  mine = warp_max_u64(mine);
  if (lane == 0) part_best[warp] = mine;
  const int any_nan = __syncthreads_or(nan);
  if (C > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");    // every block of the cluster runs
  if (warp == 0) {
    const uint64_t b = warp_max_u64(lane < kWarps ? part_best[lane] : 0ull);
    if (lane < C) { cst_u64(cluster_addr(&x_best[rank], lane), b); cst_u32(cluster_addr(&x_nan[rank], lane), any_nan ? 1u : 0u); }
  }
  cluster_sync(C);
  const uint64_t top = warp_max_u64(lane < C ? x_best[lane] : 0ull);        // every warp for itself
  const bool has_nan = __any_sync(kFull, lane < C && x_nan[lane] != 0u) != 0;
  const float vmax = best_value(top);

  // ---- the fixed-point mass relative to the maximum; the best Gumbel key and the best key that lost ---------------------------------
  const uint32_t t_id = 2000u + static_cast<uint32_t>(P.first_position + row);
  const float c2 = exp2_scale(P.temperature), inv_t32 = __double2float_rn(1.0 / static_cast<double>(P.temperature));
  uint64_t w = 0ull, key = 0ull; float second = -INFINITY;
  if (!has_nan && fabsf(vmax) < INFINITY) {
    GumbelScan g;
    g.init(seed, step, t_id, P.temperature, __fadd_rn(__fmul_rn(vmax, inv_t32), gumbel(seed, step, t_id, best_index(top))));
    draft_chunks<F32>(R, kept, [&](int c, const RawChunk<F32>& q) {
      float z[8];
      widen_raw<F32>(R, q, c, z);
      FloorSum sum;
      const int i0 = 8 * c - R.off;
      uint64_t x = g.first(i0);                                             // (the hash's arguments lie a constant apart)
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        sum.add(weight_f2(z[e], z[e + 1], vmax, c2));                       // (positions outside the row are -inf: weight 0, no key)
        g.offer2_at(canon_zero(z[e]), x, canon_zero(z[e + 1]), x + kHashStep, static_cast<uint32_t>(i0 + e));
        x += 2u * kHashStep;
      }
      w += sum.sum();
    });
    key = g.best; second = g.second;
  } else {                                                                  // a NaN, +inf, or nothing but -inf: every key, by the definition
    draft_chunks<F32>(R, kept, [&](int c, const RawChunk<F32>& q) {
      float z[8];
      widen_raw<F32>(R, q, c, z);
#pragma unroll 1
      for (int e = 0; e < 8; e++) {
        const int i = 8 * c + e - R.off;
        if (i < 0 || i >= P.vocab) continue;
        const float v = canon_zero(pick8(z, e)), k = __fadd_rn(__fmul_rn(v, inv_t32), gumbel(seed, step, t_id, static_cast<uint32_t>(i)));
        const uint64_t p = pack_best(k, static_cast<uint32_t>(i));
        if (p > key) { if (key) second = fmaxf(second, best_value(key)); key = p; } else second = fmaxf(second, k);
        w += weight_q40(v, vmax, c2);
      }
    });
  }
  const uint64_t warp_w = warp_sum_u64(w), warp_key = warp_max_u64(key);
  const float lost = key == warp_key ? second : (key ? best_value(key) : -INFINITY);   // this thread's best key that is not the warp's
  const uint32_t warp_lost = warp_max_u32(fkey(lost));
  if (lane == 0) { part_mass[warp] = warp_w; part_key[warp] = warp_key; part_rival[warp] = warp_lost; }
  __syncthreads();
  if (warp == 0) {
    const bool have = lane < kWarps;
    const uint64_t m = warp_sum_u64(have ? part_mass[lane] : 0ull), k = have ? part_key[lane] : 0ull, win = warp_max_u64(k);
    const float l = fmaxf(have ? fkey_inv(part_rival[lane]) : -INFINITY, (k && k != win) ? best_value(k) : -INFINITY);
    const uint32_t r = warp_max_u32(fkey(l));
    if (lane == 0) {
      cst_u64(cluster_addr(&x_mass[rank], 0), m);
      cst_u64(cluster_addr(&x_key[rank], 0), win);
      cst_u32(cluster_addr(&x_rival[rank], 0), __float_as_uint(fkey_inv(r)));
    }
  }
  cluster_sync(C);
  if (rank == 0 && warp == 0) {
    const bool have = lane < C;
    const uint64_t mass = warp_sum_u64(have ? x_mass[lane] : 0ull), k = have ? x_key[lane] : 0ull, win = warp_max_u64(k);
    const float edge = best_value(win) - 4e-6f;
    const bool tie = __any_sync(kFull, win && ((have && x_rival[lane] >= edge && x_rival[lane] > -INFINITY) || (k && k != win && best_value(k) >= edge))) != 0;
    if (lane == 0) {
      P.out_tokens[row] = win ? static_cast<int>(best_index(win)) : -1;
      if (P.out_vmax) P.out_vmax[row] = vmax;
      if (P.out_mass) P.out_mass[row] = mass;
      if (P.out_lse) P.out_lse[row] = mass ? __double2float_rn(static_cast<double>(vmax) / static_cast<double>(P.temperature) + log(static_cast<double>(mass) * 9.094947017729282e-13)) : -INFINITY;
      if (P.out_status) P.out_status[row] = (tie ? LM_STATUS_NEAR_TIE : 0u) | (has_nan ? LM_STATUS_NAN : 0u);
    }
  }
}

}  // namespace lm

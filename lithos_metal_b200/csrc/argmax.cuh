// Greedy argmax of every row: token = lowest index of the row's maximum, -1 for an empty row (kernels/common/argmax.metal:36-99).
//
// One launch, no workspace: a row is read by a thread-block cluster (16 blocks for a single row, one block per row once the rows fill
// the GPU), whose blocks' packed (value, lowest index) maxima meet in block 0's shared memory. (A workspace
// would have to be cleared by a memset of its own, and its atomics need a fence and a last-block test: 24 us for a single row by that way, 4 by this,
// both with the host's share.) BF16 logits are compared two at a time; per 8 logits a
// thread keeps the maximum and the chunk it lies in, and looks for its index once, at the end.
// NaN follows the packed order (a positive NaN above +inf, a negative one below -inf): a chunk that holds one is compared element by element.
#pragma once
#include <cuda_bf16.h>

#include "sample_cluster.cuh"

namespace lm {

constexpr int kArgmaxThreads = 512;

template <bool F32>
static __global__ void __launch_bounds__(kArgmaxThreads) argmax_cluster_kernel(const void* logits, int vocab, int64_t row_stride, int32_t* out32, int64_t* out64, int C) {
  __shared__ unsigned long long met[kCMaxRanks];
  __shared__ unsigned long long partial[kArgmaxThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0, row = C > 1 ? static_cast<int>(blockIdx.x) / C : static_cast<int>(blockIdx.x);
  if (C > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  after_predecessor();
  ClusterRow R;
  R.row = static_cast<const char*>(logits) + static_cast<size_t>(row) * static_cast<size_t>(row_stride) * (F32 ? 4 : 2);
  R.V = vocab; R.pen = nullptr; R.rho = 1.0f; R.pi = 0.0f; R.vals = nullptr; R.nv = 0;
  const int head = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(R.row) & 15u)) & 15u) / (F32 ? 4 : 2);
  R.off = head ? 8 - head : 0;
  const int n_chunks = (vocab + R.off + 7) / 8, per = (n_chunks + C - 1) / C;
  R.c0 = min(n_chunks, rank * per); R.c1 = min(n_chunks, R.c0 + per);
  float best = -INFINITY;
  int best_c = R.c0 + tid < R.c1 ? R.c0 + tid : -1;                         // (a row of nothing but -inf: its first element)
  uint64_t odd = 0ull;                                                      // the best of the chunks that hold a NaN
  auto take = [&](int c, const RawChunk<F32>& q) {
    float mx;
    if (F32) {
      const uint4 b = q.a[F32 ? 1 : 0];
      const uint32_t w[8] = {q.a[0].x, q.a[0].y, q.a[0].z, q.a[0].w, b.x, b.y, b.z, b.w};
      mx = __uint_as_float(w[0]);
#pragma unroll
      for (int e = 1; e < 8; e++) asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(mx), "f"(__uint_as_float(w[e])));
    } else {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q.a[0]);
      const __nv_bfloat162 m = __hmax2_nan(__hmax2_nan(h[0], h[1]), __hmax2_nan(h[2], h[3]));
      const float l = __low2float(m), r = __high2float(m);
      asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(l), "f"(r));
    }
    if (mx > best) { best = mx; best_c = c; }
    if (mx != mx) {
      float z[8];
      widen_raw<F32>(R, q, c, z);
      for (int e = 0; e < 8; e++) {
        const int i = 8 * c + e - R.off;
        if (i < 0 || i >= vocab) continue;
        const uint64_t p = pack_best(canon_zero(z[e]), static_cast<uint32_t>(i));
        odd = p > odd ? p : odd;
      }
    }
  };
  {
    constexpr int kDeep = F32 ? 2 : 4;                                      // chunks in flight per thread
    int c = R.c0 + tid;
    RawChunk<F32> q[kDeep];
#pragma unroll
    for (int j = 0; j < kDeep; j++) if (c + j * kArgmaxThreads < R.c1) q[j] = load_raw<F32>(R, c + j * kArgmaxThreads);
#pragma unroll 1
    for (; c < R.c1; c += kDeep * kArgmaxThreads) {
      RawChunk<F32> next[kDeep];
#pragma unroll
      for (int j = 0; j < kDeep; j++) { next[j] = q[j]; const int cn = c + (kDeep + j) * kArgmaxThreads; if (cn < R.c1) next[j] = load_raw<F32>(R, cn); }
#pragma unroll
      for (int j = 0; j < kDeep; j++) if (c + j * kArgmaxThreads < R.c1) take(c + j * kArgmaxThreads, q[j]);
#pragma unroll
      for (int j = 0; j < kDeep; j++) q[j] = next[j];
    }
  }
  uint64_t mine = odd;
  if (best_c >= 0) {
    const RawChunk<F32> q = load_raw<F32>(R, best_c);
    float z[8];
    widen_raw<F32>(R, q, best_c, z);
    int at = -1;
#pragma unroll
    for (int e = 7; e >= 0; e--) { const int i = 8 * best_c + e - R.off; if (z[e] == best && i >= 0 && i < vocab) at = i; }
    if (at >= 0) { const uint64_t p = pack_best(canon_zero(best), static_cast<uint32_t>(at)); mine = p > mine ? p : mine; }
  }
  mine = warp_max_u64(mine);
  if (lane == 0) partial[warp] = mine;
  __syncthreads();
  if (C > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");    // block 0 runs: its memory may be written to
  if (warp == 0) {
    mine = warp_max_u64(lane < kArgmaxThreads / 32 ? partial[lane] : 0ull);
    if (lane == 0) { if (C > 1) cst_u64(cluster_addr(&met[rank], 0), mine); else met[0] = mine; }
  }
  if (C > 1) cluster_sync(C);
  if (rank == 0 && warp == 0) {
    __syncwarp();
    const uint64_t b = warp_max_u64(lane < C ? met[lane] : 0ull);
    if (lane == 0) {
      const int token = b ? static_cast<int>(best_index(b)) : -1;
      if (out64) out64[row] = token; else out32[row] = token;
    }
  }
}

}  // namespace lm

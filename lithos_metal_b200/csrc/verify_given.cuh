// Stochastic verification given the rows' maxima and masses (what the sampler that made the thresholds knows): one logit per draft tells the decisive row, and
// every block finds it for itself. That row is all there is to draw from, so it is cut over ALL blocks, an SM each, a thread to half a chunk of eight logits;
// their shares -- the residual's, and the row's own for a residual that is empty -- are words in the workspace, and the block that arrives last chooses the share
// with the draw's point and weighs that block's slice once more for the token. (No block waits for another: a word says itself that it is this launch's.) It is
// bound by its chain: the drafts' logits, the row's slice, an arrival, the shares, the slice again. us a call in a CUDA graph, the decisive row on the 16 SMs of its
// cluster / so (7 drafts but where 15 are said; the first one rejected; 148 blocks that met by polled words in a cooperative launch in brackets): 151,936 tokens 12.1 / 8.3
// (11.9), with thresholds of top_p 0.95 19.8 / 8.5 (12.1), of top_k 50 8.9 / 7.8 (10.7), drafter's logits 12.5 / 8.3 (13.0), the reference's draw 18.0 / 9.8 (10.7), 15 drafts
// 12.9 / 8.4 (12.2); 248,320 15.0 / 8.6 (12.2), with top_p 28.5 / 8.7 (12.4); 50,257 8.5 / 8.1 (11.0); 16,384 7.7 / 7.9 (11.0): 32,000 and less
// are the only sizes to lose.
#pragma once
#include "verify.cuh"

namespace lm {

struct VerifyGivenSmem {
  VerifyRow row; int j, last, block, token; float vmax; unsigned long long mass; uint64_t left;
  uint64_t own[kVerifyWarps], res[kVerifyWarps];
};

template <bool F32, int Q>
static __global__ void __launch_bounds__(kVerifyThreads) verify_given_kernel(const __grid_constant__ VerifyDev P) {
  __shared__ VerifyGivenSmem s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = static_cast<int>(gridDim.x), V = P.vocab;
  constexpr int kSize = F32 ? 4 : 2;
  const bool gumbel = P.draw == LM_DRAW_GUMBEL;
  after_predecessor();
  unsigned long long launch;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(launch) : "l"(&P.ws->launches) : "memory");
  VerifyRound rd;
  if (!verify_begin(P, rd)) return;
  const float c2 = exp2_scale(P.temperature);
  const float u_final = P.u_final ? P.u_final[0] : 0.0f;                     // (wanted at the very end)
  // ---- the decisive row ------------------------------------------------------------------------------------------------------------------
  if (warp == 0) {
    const int r = lane & 15;
    const bool tests = r < rd.L, drafter = lane >= 16;
    VerifyTest<F32, Q> t;
    t.load(P, rd, tests, true, r);
    ProbScale scale;                                                        // (a lane's own row: the division while the logits are on their way)
    scale.init(t.mass);
    if (!drafter) t.vmax = canon_zero(t.vmax);
    const float pq = t.prob(t.vmax, t.mass, c2);
    const uint32_t rejects = __ballot_sync(kFull, t.rejects(pq) && tests && !drafter);
    if (blockIdx.x == 0 && P.out_p_draft && tests && !drafter) P.out_p_draft[r] = pq;
    const int j = rejects ? __ffs(static_cast<int>(rejects)) - 1 : rd.L;
    VerifyRow& x = s.row;
    if (lane == j) { s.j = j; s.vmax = t.vmax; s.mass = t.mass; x.tau = t.tau; x.p_of = scale; x.cut = P.tau != nullptr; x.c2 = c2; x.V = V; }
    if (Q == 2 && lane == j + 16 && tests) { x.qv = t.vmax; x.q_of = scale; }
  }
  __syncthreads();
  const int j = s.j, row = rd.row0 + j;
  const bool has_q = j < rd.L;
  const float vmax = s.vmax, tau = s.row.tau;
  const unsigned long long mass = s.mass;
  // ---- this block's slice of it ----------------------------------------------------------------------------------------------------------
  const char* z_row = static_cast<const char*>(P.target) + static_cast<size_t>(row) * static_cast<size_t>(P.row_stride) * kSize;
  const int head = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(z_row) & 15u)) & 15u) / kSize;
  const int off = head ? 8 - head : 0, n_chunks = (V + off + 7) / 8, per = (n_chunks + G - 1) / G;
  const char* q_row = !has_q ? nullptr : Q == 1 ? reinterpret_cast<const char*>(P.q + static_cast<int64_t>(j) * P.q_stride) : reinterpret_cast<const char*>(P.q_logits + static_cast<int64_t>(j) * P.q_logits_stride);
  const bool q_vec = ((reinterpret_cast<uintptr_t>(q_row) - static_cast<uintptr_t>(off) * (Q == 1 ? 4 : 2)) & 15u) == 0u;
  if (Q == 1 && lane == 0) { s.row.z_row = z_row; s.row.q_row = q_row; s.row.off = off; }   // (for verify_below_zero: every warp writes the same)
  __syncwarp();
  // Half g & 1 of chunk g >> 1: its logits, and its weights in the draw over the row itself and over the residual. Returns the latter's (of 2^40) one by one, the
  // former's where there is no draft or `own_ones`.
  auto weigh = [&](int g, uint4& z, uint64_t& own, uint64_t& res, bool own_ones) {
    const int c = g >> 1, h = g & 1, zi = 8 * c - off + (F32 ? 4 * h : 0), qi = 8 * c - off + (Q == 1 ? 4 * h : 0);
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    if (zi >= 0 && zi + (F32 ? 4 : 8) <= V) z = __ldg(reinterpret_cast<const uint4*>(z_row + static_cast<int64_t>(zi) * kSize));
    else z = verify_far<F32>(z_row, off, V, c, h, false, F32 ? 0xFF800000u : 0xFF80u);
    if (has_q) {
      if (q_vec && qi >= 0 && qi + (Q == 1 ? 4 : 8) <= V) q = __ldg(reinterpret_cast<const uint4*>(q_row + static_cast<int64_t>(qi) * (Q == 1 ? 4 : 2)));
      else q = verify_far<Q == 1>(q_row, off, V, c, h, false, Q == 1 ? 0u : 0xFF80u);
    }
    float4 x = verify_weights<F32>(s.row, z, h, vmax);
    FloorSum sum;
    const float2 a = sum.add(make_float2(x.x, x.y)), b = sum.add(make_float2(x.z, x.w));
    own = sum.sum();
    x = make_float4(a.x, a.y, b.x, b.y);
    res = 0ull;
    if (!has_q) return x;
    const float4 r = verify_rest<F32, Q>(s.row, x, q, c, h, vmax);
    FloorSum left;
    left.add(make_float2(r.x, r.y)); left.add(make_float2(r.z, r.w));
    res = left.beyond() ? verify_wide(r, make_float4(0.0f, 0.0f, 0.0f, 0.0f)) : left.sum();
    return own_ones ? x : r;
  };
  {
    const int g0 = 2 * min(n_chunks, static_cast<int>(blockIdx.x) * per), g1 = min(2 * n_chunks, g0 + 2 * per);
    uint64_t own = 0ull, res = 0ull;
    ResidualScan rest;
    GumbelScan keys;
    if (gumbel) { rest.init(rd.seed, rd.step, 4000u); keys.init(rd.seed, rd.step, static_cast<uint32_t>(row), P.temperature, -INFINITY); }
    if (mass > 0ull) {
#pragma unroll 1
      for (int g = g0 + tid; g < g1; g += kVerifyThreads) {
        uint4 z;
        uint64_t o, w;
        const float4 x = weigh(g, z, o, w, false);
        own += o; res += w;
        if (gumbel) {
          const int i = 4 * g - off;
          const float r4[4] = {x.x * 0x1p-40f, x.y * 0x1p-40f, x.z * 0x1p-40f, x.w * 0x1p-40f};
          if (has_q) rest.offer4(r4, i);
          float2 y[2];
          verify_pairs<F32>(z, g & 1, y);
#pragma unroll
          for (int k = 0; k < 2; k++)                                       // (what is not kept, or lies outside the row, is -inf: no key)
            keys.offer2(y[k].x >= tau ? y[k].x : -INFINITY, static_cast<uint32_t>(i + 2 * k), y[k].y >= tau ? y[k].y : -INFINITY, static_cast<uint32_t>(i + 2 * k + 1));
        }
      }
    }
    res = gumbel ? warp_max_u64(rest.best) : warp_sum_u64(res);
    own = gumbel ? warp_max_u64(keys.best) : warp_sum_u64(own);
    if (lane == 0) { s.res[warp] = res; s.own[warp] = own; }
  }
  // ---- the shares, and the block that arrives last --------------------------------------------------------------------------------------------
  const unsigned long long tag = (launch + 1ull) << 32;                     // (a word never written is 0)
  __syncthreads();
  if (warp == 0) {
    const uint64_t a = lane < kVerifyWarps ? s.res[lane] : 0ull, b = lane < kVerifyWarps ? s.own[lane] : 0ull;
    const uint64_t res = gumbel ? warp_max_u64(a) : warp_sum_u64(a), own = gumbel ? warp_max_u64(b) : warp_sum_u64(b), mine = lane < 2 ? res : own;
    if (lane < 4 && !(P.withhold && blockIdx.x == 0))
      asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&P.ws->part[blockIdx.x][lane]), "l"(tag | ((lane & 1) ? mine >> 32 : mine & 0xFFFFFFFFull)) : "memory");
    unsigned before = 0u;
    if (lane == 0) {
      asm volatile("atom.add.relaxed.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(&P.ws->arrived) : "memory");
      s.last = before == static_cast<unsigned>(G) - 1u;
    }
  }
  __syncthreads();
  if (!s.last) return;
  const unsigned limit = P.wait_limit ? P.wait_limit : kVerifyWaitLimit;
  bool late = false, residual = false;
  uint64_t share[2] = {0ull, 0ull};                                         // of block tid: the residual's, the row's own (or their best keys)
  if (tid < G) {
#pragma unroll 1
    for (unsigned spins = 0;; spins++) {
      unsigned long long w[4];
#pragma unroll
      for (int k = 0; k < 4; k++) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w[k]) : "l"(&P.ws->part[tid][k]) : "memory");
      share[0] = (w[0] & 0xFFFFFFFFull) | (w[1] << 32); share[1] = (w[2] & 0xFFFFFFFFull) | (w[3] << 32);
      if ((((w[0] ^ tag) | (w[1] ^ tag) | (w[2] ^ tag) | (w[3] ^ tag)) >> 32) == 0ull) break;
      if (spins >= limit) { late = true; break; }
      if (spins > 64u) __nanosleep(100);
    }
  }
  // ---- the draw ----------------------------------------------------------------------------------------------------------------------------
  // (the running sums of a warp's shares while the other warps add theirs up)
  uint64_t incl[2] = {share[0], share[1]};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t a = __shfl_up_sync(kFull, incl[0], o), b = __shfl_up_sync(kFull, incl[1], o);
    if (lane >= o) { incl[0] = gumbel ? max(incl[0], a) : incl[0] + a; incl[1] = gumbel ? max(incl[1], b) : incl[1] + b; }
  }
  if (lane == 31) { s.res[warp] = incl[0]; s.own[warp] = incl[1]; }
  if (tid == 0) { s.block = -1; s.token = -1; }
  const bool bad = __syncthreads_or(late) != 0;
  uint64_t left = 0ull;
  if (gumbel) {
    const uint64_t r = warp_max_u64(lane < kVerifyWarps ? s.res[lane] : 0ull), o = warp_max_u64(lane < kVerifyWarps ? s.own[lane] : 0ull), best = has_q && r ? r : o;
    if (tid == 0 && best) s.token = static_cast<int>(best_index(best));
  } else {
    VerifySums warps;
    const uint64_t there = verify_sums(reinterpret_cast<const unsigned long long*>(s.res), kVerifyWarps, warps);
    residual = has_q && there > 0ull;                                       // or nothing of p - q is left: the draw is over the row's own kept set
    if (!residual) verify_sums(reinterpret_cast<const unsigned long long*>(s.own), kVerifyWarps, warps);
    left = cdf_target(P.u_final ? u_final : uniform01(rd.seed, rd.step, 4000u, 0u), residual ? there : mass);
    const int at = verify_slot(warps, left);
    if (at == warp) {
      VerifySums shares{residual ? share[0] : share[1], residual ? incl[0] : incl[1]};
      const int block = verify_slot(shares, left);
      if (lane == 0) { s.block = block < 0 ? -1 : 32 * warp + block; s.left = left; }
    }
  }
  __syncthreads();
  if (s.block >= 0 && !bad) {
    // the slice with the draw's point, once more: the half by a scan over the block, the element inside it by its thread
    const int g0 = 2 * min(n_chunks, s.block * per), g1 = min(2 * n_chunks, g0 + 2 * per);
    left = s.left;
#pragma unroll 1
    for (int b0 = g0; b0 < g1; b0 += kVerifyThreads) {
      const int g = b0 + tid;
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      uint64_t sum = 0ull;
      if (g < g1) {
        uint4 z;
        uint64_t own, res;
        x = weigh(g, z, own, res, !residual);
        sum = residual ? res : own;
      }
      uint64_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
      if (lane == 31) s.own[warp] = incl;
      __syncthreads();
      VerifySums warps;
      const uint64_t total = verify_sums(reinterpret_cast<const unsigned long long*>(s.own), kVerifyWarps, warps);
      const int at = verify_slot(warps, left);
      if (at == warp && incl - sum <= left && left < incl) {
        left -= incl - sum;
        const float v[4] = {x.x, x.y, x.z, x.w};
        int token = -1;
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const uint64_t w = __float2ull_rz(v[e]);
          if (token < 0 && left < w) token = 4 * g + e - off;
          left -= w;
        }
        s.token = token;
      }
      if (at >= 0) break;
      left -= total;
      __syncthreads();                                                      // (everybody has read the warps' sums)
    }
    __syncthreads();
  }
  if (warp == 0) {
    if (lane == 0) { P.ws->arrived = 0u; P.ws->launches = launch + 1ull; }
    verify_outputs(P, rd, bad, j, s.token);
  }
}

}  // namespace lm

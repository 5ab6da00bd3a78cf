// The launches of the cluster row sampler (a translation unit of its own: it is compiled beside the others).
#include <cuda_runtime.h>

#include "argmax.cuh"
#include "draft_q.cuh"
#include "host.cuh"
#include "sample_cluster.cuh"
#include "verify_given.cuh"

namespace lm {

// Blocks per row of the argmax and the draft draw: as many as keep `slots` places busy (16 needs an opt-in), slices of at least 2048 logits.
static int cluster_blocks(int64_t rows, int64_t vocab, int slots) {
  int c = rows * 20 <= slots ? 16 : rows * 8 <= slots ? 8 : rows * 4 <= slots ? 4 : rows * 2 <= slots ? 2 : 1;
  while (c > 1 && vocab < 2048LL * c) c >>= 1;
  return c;
}

// Blocks per row of the sampler. A cluster lies within one group of 16 to 18 SMs, so with a block per SM 148 SMs hold seven clusters of 16,
// fifteen of 8 and thirty-two of 4 at once, and one row more waits for a second round (16 rows of 151,936, top_k 20: 41 us with 8 blocks
// each, 29 us with 4). Beyond that the blocks share SMs, and a row without a top_k takes several times as long as one with: smaller pieces
// even that out where the slices stay long (binary32 rows with mixed knobs, us with 1 / 2 / 4 blocks: 96 rows of 151,936 198 / 184 / 126,
// 96 of 65,536 96 / 78 / 87, 400 of 50,257 193 / 175 / 280, 400 of 24,576 119 / 136 / 243).
// `listed_k`: the top_k that every row has, with a list (0: they differ, or have none). Two blocks to a row then, but for the longest rows of 33 to 64, whose
// quarters no longer fit shared memory and so lie two to an SM, twice thirty-two clusters at once: us with 2 / 4 blocks,
//   BF16, top_k 50: 64 rows of 151,936 25.0 / 35.4, of 196,608 29.9 / 30.9, of 229,376 33.9 / 33.2, of 262,144 38.7 / 37.0; of 262,144 40 rows 34.1 / 34.9, 48 34.7 / 34.9,
//   56 37.0 / 35.0, 74 39.8 / 57.5; top_k 512: 64 rows of 196,608 38.2 / 39.0, of 245,760 44.6 / 42.9, 40 of those 39.8 / 41.0 (the line: 80,000 logits to an SM);
//   a longer list sooner: top_k 700, of 180,224 40 rows 38.6 / 39.0, 64 40.9 / 42.4, of 196,608 41.5 / 39.3 and 42.3 / 41.7; 1000, 64 rows of those 48.5 / 45.9;
//   binary32, top_k 20: of 172,032 40 rows 29.4 / 30.2, of 196,608 32.3 / 30.8, 64 35.5 / 37.0, of 229,376 39.5 / 39.6, of 262,144 42.4 / 41.1.
static int sample_blocks(int64_t rows, int64_t vocab, int sms, bool f32, int listed_k) {
  const bool listed = listed_k > 0;
  int c = 1;
  if (rows * 20 <= sms) c = 16;
  else if (rows * 48 <= 5LL * sms) c = 8;
  else if (rows * 9 <= 2LL * sms) c = 4;
  else if (!listed && rows <= 2LL * sms && vocab >= (rows * 3 <= sms ? 49152 : 98304)) c = 4;
  else if (listed && rows * 16 <= 7LL * sms && vocab >= 196608 &&
           (listed_k > 512 || (f32 ? rows * 8 <= 3LL * sms || vocab >= 229376 : vocab >= 229376 && rows * vocab >= 80000LL * sms))) c = 4;
  else if (rows * 2 <= sms) c = 2;
  else if (listed ? rows <= 2LL * sms && vocab >= 65536 : rows * 3 <= 2LL * sms || (rows <= 3LL * sms && vocab >= 40000)) c = 2;
  while (c > 1 && vocab < 2048LL * c) c >>= 1;
  return c;
}

// The instances of the sampler: FP32 / BF16 rows, the slices cached in shared memory or not, and then one block per SM or two.
constexpr size_t kAloneSmem = 116 * 1024;                                  // more than half of an SM's shared memory
constexpr size_t kMostSmem = 227 * 1024, kHalfSmem = kMostSmem / 2 - 1024;
struct ClusterPlan { int C; size_t smem; bool cached, two, ordered, few; };

template <bool F32, bool CACHED, int kPerSM>
static int cluster_ready(int instance, int C, bool* fits) {
  const void* fn = reinterpret_cast<const void*>(sample_cluster_kernel<F32, CACHED, kClusterBlock, kPerSM>);
  const KernelSlot slot = static_cast<KernelSlot>(kSlotCluster + instance);
  const size_t most = kPerSM == 2 ? kHalfSmem : kMostSmem;                  // (what any call of the instance may need: one answer for all of them)
  const int rc = ensure_dynamic_smem(slot, fn, most, true);
  *fits = rc == LM_OK && (C == 1 || cluster_fits(slot, fn, kClusterBlock, most, C));
  return rc;
}
static int cluster_ready(bool f32, const ClusterPlan& p, bool* fits) {
  if (p.cached) return f32 ? cluster_ready<true, true, 1>(0, p.C, fits) : cluster_ready<false, true, 1>(1, p.C, fits);
  if (p.two) return f32 ? cluster_ready<true, false, 2>(2, p.C, fits) : cluster_ready<false, false, 2>(3, p.C, fits);
  return f32 ? cluster_ready<true, false, 1>(4, p.C, fits) : cluster_ready<false, false, 1>(5, p.C, fits);
}

template <bool F32, bool CACHED, int kPerSM>
static int launch_cluster(const SampleDev& P, const ClusterPlan& p, cudaStream_t st) {
  return launch_beside(sample_cluster_kernel<F32, CACHED, kClusterBlock, kPerSM>, dim3(static_cast<unsigned>(P.rows) * static_cast<unsigned>(p.C)), kClusterBlock,
                       p.smem, p.C, st, P, p.C, (p.ordered ? kCallOrdered : 0u) | (p.few ? kCallFew : 0u));
}

int sample_clusters(const SampleDev& P, int sms, cudaStream_t st, bool few) {
  const bool pen = P.history != nullptr && P.hist_len > 0, f32 = P.dtype == LM_DTYPE_F32;
  const size_t head = cluster_smem_head();
  const size_t generic = sizeof(GenericSmem) + (pen ? static_cast<size_t>((P.vocab + 31) / 32) * 4 : 0) + 16;
  auto plan = [&](int C) {
    const size_t per = (static_cast<size_t>((P.vocab + 14) / 8) + C - 1) / C;    // chunks of a slice, for any alignment of the row
    const size_t marks = pen ? (per + 15) / 16 * 16 : 0;
    ClusterPlan p;
    p.C = C; p.few = few;
    p.cached = head + per * 32 + marks <= kMostSmem && C > 1;              // (a block per row reads its row from L2: two of them share an SM)
    p.smem = head + (p.cached ? per * 32 : 0) + marks;
    if (p.smem < generic) p.smem = generic;
    p.two = static_cast<long long>(P.rows) * C > sms && p.smem <= kHalfSmem;   // two blocks per SM
    p.ordered = P.top_k != nullptr && P.rows <= kOrderRows && static_cast<long long>(P.rows) * C > (p.two ? 2LL : 1LL) * sms;   // (more clusters than run at once)
    return p;
  };
  int rc = LM_OK;
  bool fits = false;
  const int most = sample_blocks(P.rows, P.vocab, sms, f32, P.top_k == nullptr && P.top_k_s <= kCListK && !(P.flags & LM_FLAG_EXACT_ONLY) ? P.top_k_s : 0);
  const int C = cluster_that_fits(most, [&](int c) { rc = cluster_ready(f32, plan(c), &fits); return fits || rc != LM_OK; });
  const ClusterPlan p = plan(C);
  if (rc == LM_OK && C == 1) rc = cluster_ready(f32, p, &fits);
  if (rc != LM_OK) return rc;
  if (p.cached) return f32 ? launch_cluster<true, true, 1>(P, p, st) : launch_cluster<false, true, 1>(P, p, st);
  if (p.two) return f32 ? launch_cluster<true, false, 2>(P, p, st) : launch_cluster<false, false, 2>(P, p, st);
  return f32 ? launch_cluster<true, false, 1>(P, p, st) : launch_cluster<false, false, 1>(P, p, st);
}

template <bool F32>
static int launch_argmax(const void* logits, int rows, int vocab, int64_t row_stride, int32_t* out32, int64_t* out64, int C, cudaStream_t st) {
  const KernelSlot slot = static_cast<KernelSlot>(kSlotArgmax + (F32 ? 1 : 0));
  const void* fn = reinterpret_cast<const void*>(argmax_cluster_kernel<F32>);
  const int rc = ensure_dynamic_smem(slot, fn, 1, true);
  if (rc != LM_OK) return rc;
  C = cluster_that_fits(C, [&](int c) { return cluster_fits(slot, fn, kArgmaxThreads, 0, c); });
  return launch_beside(argmax_cluster_kernel<F32>, dim3(static_cast<unsigned>(rows) * static_cast<unsigned>(C)), kArgmaxThreads, 0, C, st, logits, vocab, row_stride,
                       out32, out64, C);
}

int argmax_clusters(const void* logits, int dtype, int rows, int vocab, int64_t row_stride, int32_t* out32, int64_t* out64, cudaStream_t st) {
  int sms = 0;
  const int rc = sm_count(&sms);
  if (rc != LM_OK) return rc;
  const int C = cluster_blocks(rows, vocab, 2 * sms);                       // (two of these blocks share an SM easily)
  return dtype == LM_DTYPE_F32 ? launch_argmax<true>(logits, rows, vocab, row_stride, out32, out64, C, st)
                               : launch_argmax<false>(logits, rows, vocab, row_stride, out32, out64, C, st);
}

template <bool F32>
static int launch_draft_q(const DraftQDev& P, int C, int sms, cudaStream_t st) {
  const KernelSlot slot = static_cast<KernelSlot>(kSlotDraftQ + (F32 ? 1 : 0));
  const void* fn = reinterpret_cast<const void*>(draft_q_kernel<F32>);
  const int rc = ensure_dynamic_smem(slot, fn, kAloneSmem, true);
  if (rc != LM_OK) return rc;
  C = cluster_that_fits(C, [&](int c) { return cluster_fits(slot, fn, kDraftQThreads, kAloneSmem, c); });
  // A block asks for more than half of an SM's shared memory, so that no two of them lie on one while others are idle: made ready beside a predecessor they
  // pile up where that has left room (7 rows of 151,936 behind the verification of the round before: the round 40.0 us, 38.7 so; 15 rows of 248,320 68 to 70 and 62). Not
  // where all clusters would then not run at once: with a few blocks more than SMs they share some (8 rows of 151,936 12.3 us), with half as many again eight
  // blocks to a row, an SM each, are faster (11 rows 14.4 / 12.6, 14 rows of 262,144 18.5 / 17.8).
  auto at_once = [&](int c) { return clusters_at_once(slot, fn, kDraftQThreads, kAloneSmem, c) >= P.rows; };
  if (C > 1 && !at_once(C) && P.rows * C * 6 > sms * 7 && at_once(C / 2)) C /= 2;
  return launch_beside(draft_q_kernel<F32>, dim3(static_cast<unsigned>(P.rows) * static_cast<unsigned>(C)), kDraftQThreads, at_once(C) ? kAloneSmem : 0, C, st, P, C);
}

int draft_q_clusters(const DraftQDev& P, int sms, cudaStream_t st) {
  const int C = cluster_blocks(P.rows, P.vocab, 2 * sms);                   // (two of these blocks share an SM)
  return P.dtype == LM_DTYPE_F32 ? launch_draft_q<true>(P, C, sms, st) : launch_draft_q<false>(P, C, sms, st);
}

// The verification given the rows' maxima and masses: the decisive row over all the blocks that it is worth, an SM each (as the draft draw's: the two follow one
// another in a speculative round). A thread per half chunk is 256 chunks to a block; down to 64 more blocks are faster, up to some 120, beyond which their arrivals
// cost more (us, first of 7 drafts rejected, 48 / 80 / 120 / 148 blocks: 151,936 tokens 8.84 / 8.62 / 8.31 / 9.14, 100,000 8.63 / 8.23 / 8.22 / -, 50,257 8.75 / 8.22 / 8.08 / 8.45).
template <bool F32, int Q>
static int launch_verify_given(const VerifyDev& P, int sms, cudaStream_t st) {
  const KernelSlot slot = static_cast<KernelSlot>(kSlotVerifyGiven + (F32 ? 2 : 0) + Q - 1);
  const int rc = ensure_dynamic_smem(slot, reinterpret_cast<const void*>(verify_given_kernel<F32, Q>), kAloneSmem);
  if (rc != LM_OK) return rc;
  const int chunks = P.vocab / 8 + 1, least = (chunks + 255) / 256, most = sms < kVerifyParts ? sms : kVerifyParts;
  int grid = (chunks + 63) / 64;
  if (grid > 120) grid = least > 120 ? least : 120;
  if (grid > most) grid = most;
  return launch_stream(true, verify_given_kernel<F32, Q>, dim3(static_cast<unsigned>(grid)), kVerifyThreads, kAloneSmem, 1, st, P);
}

// ... and not given: a cluster per target row, as many blocks each as let all of them run at once. In two launches, the first of them clusters for the maxima and
// masses, where a slice does not fit shared memory (us by clusters alone / so, and by all SMs for the decisive row in a cooperative launch; first draft rejected and, in
// brackets, all accepted: 15 drafts, 200,000 tokens 53.5 / 25.5, 32.5 (27.9 / 24.8, 24.8), the reference's draw 81.3 / 27.2, 29.4; 262,144 60.5 / 27.3, 42.2; 7 drafts, 400,000
// 45.7 / 26.3, 28.9; but 3 of 1,000,000 85 / 35, 34 (40 / 35, 28)). And for the reference's draw from eight rows on, whose eighth cluster of sixteen shares another's SMs, where
// rows are long (7 drafts, 151,936 tokens 23.6 / 17.3, 21.2 (14.8 / 15.3, 19.7), 65,536 15.4 / 14.6, 20.5 (10.9 / 13.0, 19.9); 15 of 100,000 27.6 / 17.8, 24.3 (18.4 / 16.2, 25.7);
// 3 of 151,936 16.9 / 17.1, 17.6 (13.7 / 15.2, 16.7)).
template <bool F32, int Q, int kMode>
static int launch_verify(const VerifyDev& P, int sms, cudaStream_t st) {
  const KernelSlot slot = static_cast<KernelSlot>(kSlotVerify + (F32 ? 6 : 0) + (Q == 0 ? 0 : kMode == kVerifyStats ? 1 : 2 * Q + kMode));
  const void* fn = reinterpret_cast<const void*>(verify_kernel<F32, Q, kMode>);
  const int rc = ensure_dynamic_smem(slot, fn, kVerifySmem, true);
  if (rc != LM_OK) return rc;
  const int rows = P.n_draft + 1;
  const int C = cluster_that_fits(cluster_blocks(rows, P.vocab, 2 * sms), [&](int c) { return clusters_at_once(slot, fn, kVerifyThreads, kVerifySmem, c) >= rows; });
  const size_t chunks = (static_cast<size_t>((P.vocab + 14) / 8) + C - 1) / C;   // of a slice, for any alignment of the row
  const size_t z = chunks * 32 + (chunks + 1) / 2 * 16, q = Q == 0 || kMode == kVerifyStats ? 0 : chunks * 32;   // (logits, then weights; the chunks' sums; the drafter's row, then the residual's weights)
  const bool z_cached = z <= kVerifySmem, q_cached = q != 0 && (z_cached ? z : 0) + q <= kVerifySmem;
  if (Q != 0 && kMode != kVerifyStats && (!z_cached || (kMode == kVerifyNoise && rows * 20 > sms && P.vocab >= 98304))) {
    const int rc1 = launch_verify<F32, 1, kVerifyStats>(P, sms, st);
    if (rc1 != LM_OK) return rc1;
    VerifyDev G = P;
    G.row_max = P.ws->vmax; G.row_mass = P.ws->mass;
    return launch_verify_given<F32, Q == 0 ? 1 : Q>(G, sms, st);
  }
  const size_t smem = (z_cached ? z : 0) + (q_cached ? q : 0);
  const unsigned grid = static_cast<unsigned>(rows) * static_cast<unsigned>(C);
  return launch_stream(static_cast<int>(grid) <= sms, verify_kernel<F32, Q, kMode>, dim3(grid), kVerifyThreads, smem, C, st, P, C, z_cached ? 1 : 0, q_cached ? 1 : 0);
}

template <bool F32>
static int launch_verify_rows(const VerifyDev& P, int sms, cudaStream_t st) {
  if (P.mode != LM_VERIFY_STOCHASTIC) return launch_verify<F32, 0, kVerifyDraw>(P, sms, st);
  if (P.row_max && P.row_mass) return P.q ? launch_verify_given<F32, 1>(P, sms, st) : launch_verify_given<F32, 2>(P, sms, st);
  if (P.draw == LM_DRAW_GUMBEL) return P.q ? launch_verify<F32, 1, kVerifyNoise>(P, sms, st) : launch_verify<F32, 2, kVerifyNoise>(P, sms, st);
  return P.q ? launch_verify<F32, 1, kVerifyDraw>(P, sms, st) : launch_verify<F32, 2, kVerifyDraw>(P, sms, st);
}

int verify_rows(const VerifyDev& P, int sms, cudaStream_t st) {
  return P.dtype == LM_DTYPE_F32 ? launch_verify_rows<true>(P, sms, st) : launch_verify_rows<false>(P, sms, st);
}

}  // namespace lm

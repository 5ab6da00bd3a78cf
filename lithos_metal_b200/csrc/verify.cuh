// DSpark verification of one speculative step, in one launch but for the largest rows: up to n_draft drafted tokens against n_draft + 1 rows of target
// logits. Greedy: row-wise argmax and prefix match (kernels/common/spec_ops.metal:162-165). Stochastic: accept draft r with
// probability min(1, p/q), replace the first rejected one by a draw from max(p - q, 0) (kernels/common/sample.metal:273-347),
// on the integer fixed-point weights so the outcome is independent of how the vocabulary is split between blocks.
//
// The step is latency-bound (a few MB of input and a chain of dependencies: row maximum -> row mass and accept test -> the
// residual's total -> the token). A row's chain is its own business but for one bit, whether its draft is accepted. So every target row has a
// thread-block CLUSTER (16 blocks for up to 14 rows, 8 beyond, fewer where slices would be below 2048 logits or the device cannot hold them all): its slices of the row and of the drafter's row land in shared memory by asynchronous
// copies, all in flight at once; the blocks meet in distributed shared memory, a cluster barrier to a dependency; and every row that could be the
// decisive one -- its own draft rejected, or the bonus row -- draws its token without waiting for the rows before it. What a row found is one word in
// the workspace; the cluster that arrives last picks the first rejected row and writes the outputs, so no block waits for another cluster.
// A launch that is given the rows' maxima and masses knows the decisive row from one logit per draft: verify_given.cuh. Rows whose slices do not fit shared memory
// have their maxima and masses found by clusters and go on there in a second launch, and so does the reference's draw of long rows whose clusters share SMs.
// (All rows cut over all 148 SMs by a cooperative launch, partial results exchanged as polled words in L2, three trips for the step of 7 drafts; us a call so /
// by clusters, first draft rejected: V = 151,936, drafter's probabilities 20.9 / 14.7, given the maxima 19.8 / 13.0, drafter's logits 23.2 / 15.1, greedy 8.6 / 7.8; 15
// drafts 27 / 22.7; 50,257 22 / 10.8; 248,320 26 / 16.6. A cooperative launch of the clusters is not made ready beside its predecessor: 1.1 us more.)
//
// A word carries the launch's number, which the last cluster counts up: were one missing, the wait for it is bounded, and the launch reports an error through
// its outputs (and through the StepState when it commits); the GPU is never left waiting.
//
// With a StepState given, the kernel takes the round from it on the device, as the reference's kernels do
// (kernels/common/sample.metal:283-296): verify length, drafts (pending_tokens), seed, step, and it leaves at once when the
// state is done. The accept uniforms then come from the reference's stream 3000 + r of the counter-based noise.
#pragma once
#include "sample_cluster.cuh"
#include "spec_ops.cuh"

namespace lm {

constexpr int kVerifyThreads = 512;
constexpr int kVerifyWarps = kVerifyThreads / 32;
constexpr int kVerifyMaxRows = LM_MAX_DRAFT + 1;
constexpr unsigned kVerifyWaitLimit = 1u << 17;         // polls of one word before the last cluster gives up: about 0.1 s
constexpr int kVerifyParts = 256;                       // most blocks that share a row (verify_given.cuh)
// Most shared memory of a block (two to an SM). A chunk of eight logits takes 40 bytes of it (logits, then weights, in binary32; their sum), 32 more where the
// drafter's row lies there too: both do up to 1564 chunks a block, the target's alone up to 2816 (16 blocks: 200,200 and 360,400 logits).
constexpr size_t kVerifySmem = 110 * 1024;

struct VerifyWs {                                       // lives in the caller's workspace, zero-filled once
  unsigned long long launches;                          // so far
  unsigned arrived, pad;                                // rows (or, of a launch that cuts one row, blocks) of this launch that have been through (0 between launches)
  unsigned long long row[kVerifyMaxRows];               // what a row's cluster found: launch number << 24 | kFound | rejected << 21 | token + 1
  unsigned long long mass[kVerifyMaxRows];               // rows' masses and maxima, by row of the step, from a launch that finds nothing else to the one behind it
  float vmax[kVerifyMaxRows];
  unsigned long long part[kVerifyParts][4];             // a block's shares (verify_given.cuh), in halves: launch number + 1 << 32 | half
};
constexpr unsigned long long kFound = 1ull << 22, kRejected = 1ull << 21;
static_assert(LM_MAX_VOCAB < (1 << 21), "a token and 'none' fit 21 bits");

struct VerifyDev {
  int mode; int dtype; int n_draft; int vocab; int64_t row_stride; int draw;
  const void* target; const int32_t* drafts; const float* q; int64_t q_stride; float temperature;
  const uint16_t* q_logits; int64_t q_logits_stride; const float* q_vmax; const unsigned long long* q_mass;   // q from the drafter's BF16 logits when q is null
  const float* tau; const float* u_accept; const float* u_final;
  const float* row_max;                                  // stochastic mode, optional: the exact maxima of the step's rows (from the sampler): spares the first exchange
  const unsigned long long* row_mass;                    // ... and their kept sets' fixed-point masses (needs row_max): the decisive row is known at once
  uint64_t seed; uint32_t step;
  int32_t* out_accept; int32_t* out_final; int32_t* out_tokens; float* out_p_draft;
  VerifyWs* ws;
  uint32_t* state; int t_max, g;                          // StepState (optional): the round is read from it
  int commit; AcceptDev accept;                          // commit != 0: close the round on the StepState as accept_scan would
  unsigned wait_limit; unsigned withhold;                // self-test of the bounded wait: the first row's cluster does not say what it found
};

// The binary32 probabilities of weights: fl32(double(w) / double(k)) (prob_q40), two at a time and without FP64. A weight is a binary32 value; 1 / k is split in two of
// them, so that w * 1 / k is a sum p0 + p1 that is off by less than 2^-46 of it (the product's rounding is taken along by a multiply-add). Where p0 + p1 rounds
// to the same binary32 with 2^-44 more and less, every value in between does, the quotient and its FP64 rounding among them; else (one in half a million) FP64
// decides. Nothing is subnormal: w >= 1 or 0, k < 2^64.
struct ProbScale {
  float hi, lo; unsigned long long k;
  __device__ __forceinline__ void init(unsigned long long mass) {
    k = mass;
    const double inv = mass ? 1.0 / __ull2double_rn(mass) : 0.0;
    hi = __double2float_rn(inv); lo = __double2float_rn(inv - static_cast<double>(hi));
  }
  static __device__ __noinline__ float exact(float w, unsigned long long k) { return __double2float_rn(__ddiv_rn(static_cast<double>(w), __ull2double_rn(k))); }
  __device__ __forceinline__ float2 of(float2 w) const {
    const float2 h = make_float2(hi, hi), l = make_float2(lo, lo);
    const float2 p0 = __fmul2_rn(w, h), p1 = __ffma2_rn(w, l, __ffma2_rn(w, h, make_float2(-p0.x, -p0.y)));
    float2 a = __fadd2_rn(p0, __ffma2_rn(p0, make_float2(0x1p-44f, 0x1p-44f), p1));
    const float2 b = __fadd2_rn(p0, __ffma2_rn(p0, make_float2(-0x1p-44f, -0x1p-44f), p1));
    if (a.x != b.x) a.x = exact(w.x, k);
    if (a.y != b.y) a.y = exact(w.y, k);
    return a;
  }
};

// The round's bookkeeping, by the warp whose lane 0 has just written out_tokens: the accept scan on those tokens
// (kernels/common/spec_ops.metal:148-195). A prefill chunk takes the scan's prefill branch, which reads no token. All 32 lanes call.
static __device__ __noinline__ void verify_commit(const VerifyDev& P, bool failed) {
  if (!P.commit) return;
  __syncwarp();
  StepStateView st{P.accept.state, P.accept.t_max, P.accept.g};
  if (st.done()) return;
  if (failed) { if ((threadIdx.x & 31) == 0) fail_state(st, kErrBarrier); return; }   // a wait of this launch ran out: nothing to commit
  if (!P.state && st.prefill_left() == 0u && (st.verify_len() != static_cast<uint32_t>(P.n_draft) || st.t_this_step() != static_cast<uint32_t>(P.n_draft) + 1u)) {
    if ((threadIdx.x & 31) == 0) fail_state(st, kErrRoundMismatch);        // the round came from the arguments and the state describes another
    return;
  }
  __threadfence();
  round_close(P.accept);
}

// What a launch verifies: from its arguments, or from the StepState.
struct VerifyRound { int L, row0; uint64_t seed; uint32_t step; };
// False: nothing is verified, as the state is done, this step is a prefill chunk (block 0 still closes it: the scan's prefill branch), or the state's rows do not fit
// the launch (block 0 reports the caller's error).
// closes: this launch does that.
__device__ __forceinline__ bool verify_begin(const VerifyDev& P, VerifyRound& rd, bool closes = true) {
  rd = VerifyRound{P.n_draft, 0, P.seed, P.step};
  if (!P.state) return true;
  StepStateView st{P.state, P.t_max, P.g};
  rd.seed = st.seed(); rd.step = st.step();
  const bool first = closes && blockIdx.x == 0 && threadIdx.x < 32;
  if (st.done()) return false;
  if (st.prefill_left() > 0u) {
    if (first) verify_commit(P, false);
    return false;
  }
  const uint32_t len = st.verify_len(), rows = st.t_this_step();
  if (len > static_cast<uint32_t>(P.n_draft) || rows < len + 1u || rows > static_cast<uint32_t>(P.n_draft) + 1u) {
    if (first && threadIdx.x == 0) { P.out_accept[0] = -1; P.out_final[0] = -1; fail_state(st, kErrRoundMismatch); }
    return false;
  }
  rd.L = static_cast<int>(len); rd.row0 = static_cast<int>(rows - 1u - len);
  return true;
}

__device__ __forceinline__ int verify_draft(const VerifyDev& P, const VerifyRound& rd, int r) {
  return P.state ? StepStateView{P.state, P.t_max, P.g}.pending(rd.row0 + r + 1) : P.drafts[r];
}

// The outputs, by one warp, and the round closed on them.
static __device__ __noinline__ void verify_outputs(const VerifyDev& P, const VerifyRound& rd, bool bad, int accept, int token) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) { P.out_accept[0] = bad ? -1 : accept; P.out_final[0] = bad ? -1 : token; }
  if (P.out_tokens && lane <= rd.L) P.out_tokens[rd.row0 + lane] = bad ? -1 : (lane < accept ? verify_draft(P, rd, lane) : (lane == accept ? token : -1));
  verify_commit(P, bad);
}

// A row is through (one warp of its cluster): what it found, and if it is the last of the launch the outputs.
static __device__ __noinline__ void verify_arrive(const VerifyDev& P, const VerifyRound& rd, int r, unsigned long long launch, bool rejected, int token) {
  const int lane = threadIdx.x & 31;
  VerifyWs* ws = P.ws;
  unsigned before = 0u;
  if (lane == 0) {
    if (!(P.withhold && r == 0))
      asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&ws->row[r]),
                   "l"((launch << 24) | kFound | (rejected ? kRejected : 0ull) | static_cast<unsigned long long>(static_cast<uint32_t>(token + 1))) : "memory");
    asm volatile("atom.add.relaxed.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(&ws->arrived) : "memory");
  }
  if (__shfl_sync(kFull, before, 0) != static_cast<unsigned>(rd.L)) return;
  // every row of the launch has been through: a lane per row (a word says itself that it is there, so nothing has to be ordered by fences: they cost 1.3 us)
  const unsigned limit = P.wait_limit ? P.wait_limit : kVerifyWaitLimit;
  unsigned long long word = 0ull;
  bool late = false;
  if (lane <= rd.L) for (unsigned spins = 0;; spins++) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(word) : "l"(&ws->row[lane]) : "memory");
    if ((word >> 24) == launch && (word & kFound)) break;
    if (spins >= limit) { late = true; break; }
    if (spins > 64u) __nanosleep(100);
  }
  const bool bad = __any_sync(kFull, late) != 0;
  const uint32_t rejects = __ballot_sync(kFull, lane < rd.L && (word & kRejected));
  const int j = rejects ? __ffs(static_cast<int>(rejects)) - 1 : rd.L;
  const int drawn = __shfl_sync(kFull, static_cast<int>(word & (kRejected - 1ull)) - 1, j);
  if (lane == 0) { ws->arrived = 0u; ws->launches = launch + 1ull; }
  verify_outputs(P, rd, bad, j, drawn);
}

// Half h (four elements) of chunk c of a binary32 row, the whole chunk of a BF16 row, from global memory: rows that do not fit shared memory, and first or last
// chunks. Positions outside the row: -inf of a target row, nothing of a drafter's.
template <bool F32>
static __device__ __noinline__ uint4 verify_far(const char* row, int off, int V, int c, int h, bool vec, uint32_t outside) {
  const int base = 8 * c - off + (F32 ? 4 * h : 0);
  if (vec && base >= 0 && base + (F32 ? 4 : 8) <= V) return __ldg(reinterpret_cast<const uint4*>(row + static_cast<int64_t>(base) * (F32 ? 4 : 2)));
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    auto at = [&](int i) {
      if (i < 0 || i >= V) return outside;
      return F32 ? __ldg(reinterpret_cast<const uint32_t*>(row) + i) : static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(row) + i));
    };
    w[k] = F32 ? at(base + k) : at(base + 2 * k) | (at(base + 2 * k + 1) << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// What a row's chunks are weighed with; kept in shared memory for the functions below.
struct VerifyRow {
  const char *z_row, *q_row; int off, V; bool cut; float c2, tau, qv; ProbScale p_of, q_of;
};
struct VerifySmem {
  unsigned long long x_best[kCMaxRanks], x_own[kCMaxRanks], x_res[kCMaxRanks];   // what the blocks of the cluster leave in one another's copy
  uint64_t best[kVerifyWarps], own[kVerifyWarps], res[kVerifyWarps];             // this block's, per warp
  VerifyRow row; uint64_t own_block; bool reject;
};

// The logits of half h of a chunk in pairs (v: the half of a binary32 row, the chunk of a BF16 row), -0 as +0; -inf outside the row.
template <bool F32>
__device__ __forceinline__ void verify_pairs(uint4 v, int h, float2 (&z)[2]) {
  if (F32) { z[0] = make_float2(__uint_as_float(v.x), __uint_as_float(v.y)); z[1] = make_float2(__uint_as_float(v.z), __uint_as_float(v.w)); }
  else {
    const uint32_t a = h ? v.z : v.x, b = h ? v.w : v.y;
    z[0] = make_float2(bf16_lo(a), bf16_hi(a)); z[1] = make_float2(bf16_lo(b), bf16_hi(b));
  }
#pragma unroll
  for (int k = 0; k < 2; k++) z[k] = __fadd2_rn(z[k], make_float2(0.0f, 0.0f));
}

// The residual of half a chunk by the definition, from global memory: where the drafter's values are below 0, p - q may exceed 1, and a kept logit of weight 0 has one.
template <bool F32>
static __device__ __noinline__ float4 verify_below_zero(const VerifyRow& x, int c, int h, float vmax) {
  const float* q = reinterpret_cast<const float*>(x.q_row);
  float r[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int i = 8 * c + 4 * h + e - x.off;
    r[e] = 0.0f;
    if (i < 0 || i >= x.V) continue;
    const float z = canon_zero(F32 ? __ldg(reinterpret_cast<const float*>(x.z_row) + i) : bf16_lo(__ldg(reinterpret_cast<const uint16_t*>(x.z_row) + i)));
    if (z >= x.tau) r[e] = fmaxf(__fsub_rn(prob_q40(weight_q40(z, vmax, x.c2), x.p_of.k), __ldg(q + i)), 0.0f) * 1099511627776.0f;
  }
  return make_float4(r[0], r[1], r[2], r[3]);
}

// What half a chunk weighs, before the floors: the kept set's weights (what lies outside the row is -inf: 0). v: the half as it lies in the row. (By clusters
// for slices that do not fit shared memory.)
template <bool F32>
static __device__ __noinline__ float4 verify_weights(const VerifyRow& x, uint4 v, int h, float vmax) {
  float2 z[2], w[2];
  verify_pairs<F32>(v, h, z);
  const float tau = x.tau, c2 = x.c2;
  if (x.cut && !(fmaxf(fmaxf(z[0].x, z[0].y), fmaxf(z[1].x, z[1].y)) >= tau)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const float2 y = weight_f2(z[k].x, z[k].y, vmax, c2);
    w[k] = make_float2(z[k].x >= tau ? y.x : 0.0f, z[k].y >= tau ? y.y : 0.0f);
  }
  return make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
}
// What max(p - q, 0) leaves of a half's weights f, floors (what is not kept has weight 0, hence p = 0 and nothing left), of 2^40 and before the floors. qr: the half
// as it lies in the drafter's row.
template <bool F32, int Q>
static __device__ __noinline__ float4 verify_rest(const VerifyRow& x, float4 f, uint4 qr, int c, int h, float vmax) {
  float2 w[2] = {make_float2(f.x, f.y), make_float2(f.z, f.w)}, q[2];
  if (Q == 1) {
    q[0] = make_float2(__uint_as_float(qr.x), __uint_as_float(qr.y)); q[1] = make_float2(__uint_as_float(qr.z), __uint_as_float(qr.w));
    if (fminf(fminf(q[0].x, q[0].y), fminf(q[1].x, q[1].y)) < 0.0f) return verify_below_zero<F32>(x, c, h, vmax);
  }
  if (!(__float_as_uint(f.x) | __float_as_uint(f.y) | __float_as_uint(f.z) | __float_as_uint(f.w))) return f;
  if (Q == 2) {
    uint2 t, l;
    verify_pairs<false>(qr, h, q);
    const ProbScale q_of = x.q_of;
#pragma unroll
    for (int k = 0; k < 2; k++) q[k] = q_of.of(floor2(weight_f2(q[k].x, q[k].y, x.qv, x.c2), t, l));
  }
  const ProbScale p_of = x.p_of;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const float2 d = __fadd2_rn(p_of.of(w[k]), make_float2(-q[k].x, -q[k].y));
    w[k] = __fmul2_rn(make_float2(w[k].x > 0.0f ? fmaxf(d.x, 0.0f) : 0.0f, w[k].y > 0.0f ? fmaxf(d.y, 0.0f) : 0.0f), make_float2(1099511627776.0f, 1099511627776.0f));
  }
  return make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
}
// The floors' sum of residuals some of which may be above 2^40.
static __device__ __noinline__ uint64_t verify_wide(float4 a, float4 b) {
  return __float2ull_rz(a.x) + __float2ull_rz(a.y) + __float2ull_rz(a.z) + __float2ull_rz(a.w) + __float2ull_rz(b.x) + __float2ull_rz(b.y) + __float2ull_rz(b.z) + __float2ull_rz(b.w);
}

// Every warp for itself: the slots' running sums, a lane per slot, and their sum.
struct VerifySums { uint64_t mine, incl; };
__device__ __forceinline__ uint64_t verify_sums(const unsigned long long* slots, int n, VerifySums& v) {
  const int lane = threadIdx.x & 31;
  v.incl = v.mine = lane < n ? slots[lane] : 0ull;
#pragma unroll
  for (int o = 1; o < kCMaxRanks; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, v.incl, o); if (lane >= o) v.incl += t; }
  return __shfl_sync(kFull, v.incl, kCMaxRanks - 1);
}
// The slot in which the running sum passes `left`, which then counts from that slot's start; -1: none. It is one slot at most, the same for whoever asks, whatever
// the sums are: masses that are not the rows' can make them pass 2^64, and then more than one slot, or none, would hold the point.
__device__ __forceinline__ int verify_slot(const VerifySums& v, uint64_t& left) {
  const uint32_t hit = __ballot_sync(kFull, v.incl - v.mine <= left && left < v.incl);
  const int at = __ffs(static_cast<int>(hit)) - 1;
  left -= __shfl_sync(kFull, v.incl - v.mine, at < 0 ? 0 : at);
  return at;
}
static_assert(kVerifyWarps <= kCMaxRanks && kCMaxRanks <= 32, "slots of ranks and of warps alike, a lane each");

// The accept test of one draft, by two lanes of one warp: the target's side in lane r (or 0), the drafter's 16 lanes on.
template <bool F32, int Q>
struct VerifyTest {
  float u, tau, vmax; unsigned long long mass; uint32_t bits; bool in;       // (bits as they come: nothing waits for them before the test)
  // on: this lane has a side of row r's test. given: the target's side with the row's maximum and mass from the caller.
  __device__ __forceinline__ void load(const VerifyDev& P, const VerifyRound& rd, bool on, bool given, int r) {
    const bool drafter = (threadIdx.x & 16u) != 0u;
    constexpr int kSize = F32 ? 4 : 2;
    u = vmax = 0.0f; tau = -INFINITY; mass = 0ull; bits = 0u; in = false;
    if (given && !drafter && r <= rd.L) { vmax = P.row_max[rd.row0 + r]; mass = P.row_mass[rd.row0 + r]; if (P.tau) tau = P.tau[rd.row0 + r]; }   // (the bonus row's too)
    if (!on) return;
    const int d = verify_draft(P, rd, r);
    if (!drafter) { if (P.tau && !given) tau = P.tau[rd.row0 + r]; }
    else {
      u = P.u_accept ? P.u_accept[r] : uniform01(rd.seed, rd.step, 3000u + static_cast<uint32_t>(r), 0u);
      if (Q == 2) { vmax = __ldg(P.q_vmax + r); mass = __ldg(P.q_mass + r); }
    }
    in = d >= 0 && d < P.vocab;
    if (!in) return;
    if (!drafter) {
      const char* zp = static_cast<const char*>(P.target) + (static_cast<int64_t>(rd.row0 + r) * P.row_stride + d) * kSize;
      bits = F32 ? __ldg(reinterpret_cast<const uint32_t*>(zp)) : static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(zp))) << 16;
    } else if (Q == 1) bits = __float_as_uint(__ldg(P.q + static_cast<int64_t>(r) * P.q_stride + d));
    else bits = static_cast<uint32_t>(__ldg(P.q_logits + static_cast<int64_t>(r) * P.q_logits_stride + d)) << 16;
  }
  // p and q of the draft, side by side: a lane's probability of its logit (0 for an id outside the vocabulary)
  __device__ __forceinline__ float prob(float top, unsigned long long m, float c2) const {
    const float z = canon_zero(__uint_as_float(bits));
    return in && m > 0ull ? prob_q40(z >= tau ? weight_q40(z, top, c2) : 0ull, m) : 0.0f;
  }
  // for the target's lanes: rejected? pq: the lanes' own probabilities
  __device__ __forceinline__ bool rejects(float pq) const {
    return __shfl_down_sync(kFull, __fmul_rn(u, Q == 1 ? __uint_as_float(bits) : pq), 16) >= pq;   // (bits of an id outside the vocabulary: 0)
  }
};

// The best key of the reference's draws in a block's slice (chunks w0 .. w1 are the warp's; zs: in shared memory, the residual, or the logits of a row without a
// draft): over what is left of p - q, `weight` of it (of 2^40) in the warp's range, or over the row itself. A key of ln(the slice's weight) - 2 is missed once in
// 1600, and leaves seven or eight logits of the slice to look at closely; where none has reached that bar, it is what has been found, or none. (A bar for each warp's
// range leaves as many of every range, and a row without a bar a record a step at first; us a call of 7 drafts, 151,936 tokens, all of them rejected 26.4 / 25.6 so,
// accepted 16.6 / 15.8.)
template <bool F32>
static __device__ __noinline__ uint64_t verify_best_key(const VerifyDev& P, const VerifyRound& rd, VerifySmem& s, const uint4* zs, int w0, int w1, int per, int row, bool residual, bool has_q,
                                                        uint64_t weight, float vmax) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, off = s.row.off;
  const float tau = s.row.tau;
  if (lane == 0) s.res[warp] = weight;
  __syncthreads();
  const uint64_t there = residual ? warp_sum_u64(lane < kVerifyWarps ? s.res[lane] : 0ull) : s.own_block;
  ResidualScan rest;
  GumbelScan own;
  rest.init(rd.seed, rd.step, 4000u);
  own.init(rd.seed, rd.step, static_cast<uint32_t>(row), P.temperature, -INFINITY);
  // (Floors that add up to nothing leave residuals below 2^-40, which have their keys all the same: no bar.)
  float bar = there ? logf(__ull2float_rn(there) * 0x1p-40f) - 2.0f + (residual ? 0.0f : vmax * own.inv_t32) : -INFINITY;
  if (!(fabsf(bar) < 1e30f)) bar = -INFINITY;
#pragma unroll 1
  for (;;) {
    rest.room = 8388608.0f * ex2_approx((2e-3f - bar) * 1.44269504f);
    own.kb = INFINITY;
    own.raise(bar);
#pragma unroll 1
    for (int b0 = 2 * w0; b0 < 2 * w1; b0 = (b0 & 1) ? b0 + 63 : b0 + 1) {  // (whole warps)
      const int c = (b0 >> 1) + lane, h = b0 & 1, i = 8 * c + 4 * h - off;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (residual) {
        if (c < w1) v = zs[(h ? per : 0) + c];
        const float r4[4] = {__uint_as_float(v.x) * 0x1p-40f, __uint_as_float(v.y) * 0x1p-40f, __uint_as_float(v.z) * 0x1p-40f, __uint_as_float(v.w) * 0x1p-40f};   // p - q, exactly
        const uint64_t had = rest.best;
        rest.offer4(r4, i);
        rest.share(had);
      } else {
        float2 z[2] = {make_float2(-INFINITY, -INFINITY), make_float2(-INFINITY, -INFINITY)};
        if (c < w1) verify_pairs<F32>(!has_q ? zs[(F32 && h ? per : 0) + c] : verify_far<F32>(s.row.z_row, off, s.row.V, c, h, true, F32 ? 0xFF800000u : 0xFF80u), h, z);
        const uint64_t had = own.best;
#pragma unroll
        for (int k = 0; k < 2; k++)                                         // (what is not kept, or lies outside the row, is -inf: no key)
          own.offer2(z[k].x >= tau ? z[k].x : -INFINITY, static_cast<uint32_t>(i + 2 * k), z[k].y >= tau ? z[k].y : -INFINITY, static_cast<uint32_t>(i + 2 * k + 1));
        if (__any_sync(kFull, own.best != had)) own.raise(best_value(warp_max_u64(own.best)));
      }
    }
    const uint64_t mine = warp_max_u64(residual ? rest.best : own.best);
    if (lane == 0) s.best[warp] = mine;
    __syncthreads();
    const uint64_t top = warp_max_u64(lane < kVerifyWarps ? s.best[lane] : 0ull);
    if (bar == -INFINITY || (top && best_value(top) >= bar)) return top;
    bar = top ? best_value(top) : -INFINITY;
    __syncthreads();                                                        // (everybody has read the warps' best)
  }
}

// What a launch draws from: kVerifyDraw by inverse CDF, kVerifyNoise the reference's form, kVerifyStats nothing: it leaves the rows' maxima and masses in the workspace.
constexpr int kVerifyDraw = 0, kVerifyNoise = 1, kVerifyStats = 2;

// One row by one cluster. Q: 0 greedy, 1 the drafter's probabilities, 2 its BF16 logits and their statistics. Every part of this runs a few times a launch, so
// code that is not in the instruction cache costs as much as what it computes: a loop's chunk is unrolled, loops are not, what has been computed is kept rather
// than computed by a second copy of the code (the token was found in 2.5 to 3.3 us so, in 1 with the draw's weights kept), and the rare is in functions of its own.
template <bool F32, int Q, int kMode>
__device__ __forceinline__ void verify_row(const VerifyDev& P, const VerifyRound& rd, int r, int rank, int C, unsigned long long launch, bool z_cached, bool q_cached,
                                           uint4* zs, VerifySmem& s) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kSize = F32 ? 4 : 2;
  constexpr bool kGumbel = kMode == kVerifyNoise, kStats = kMode == kVerifyStats;
  if (Q != 0 && !kStats) z_cached = true;                                   // (else the launch is cut in two: launch_verify)
  const int V = P.vocab, L = rd.L, row = rd.row0 + r;
  const bool has_q = Q != 0 && !kStats && r < L;
  const bool given_max = Q != 0 && P.row_max != nullptr;
  // ---- this block's slice in chunks of eight; a warp's are consecutive, so that what a warp holds is a range of the row ------------------------
  const char* z_row = static_cast<const char*>(P.target) + static_cast<size_t>(row) * static_cast<size_t>(P.row_stride) * kSize;
  const int head = static_cast<int>((16u - (reinterpret_cast<uintptr_t>(z_row) & 15u)) & 15u) / kSize;
  const int off = head ? 8 - head : 0, n_chunks = (V + off + 7) / 8, per = (n_chunks + C - 1) / C;
  const int c0 = min(n_chunks, rank * per), c1 = min(n_chunks, c0 + per);
  const int cpw = ((per + kVerifyWarps - 1) / kVerifyWarps + 7) & ~7;
  const int w0 = min(c1, c0 + warp * cpw), w1 = min(c1, w0 + cpw);
  // z_cached: a chunk's logits, later the floors of its weights, in two halves; what the chunk weighs in the draw. q_cached: the drafter's row, later the
  // residual's weights.
  unsigned long long* sums = reinterpret_cast<unsigned long long*>(zs + 2 * per) - c0;
  uint4* qs = zs + (z_cached ? 2 * per + (per + 1) / 2 : 0) - c0;
  zs -= c0;
  const char* q_row = !has_q ? nullptr : Q == 1 ? reinterpret_cast<const char*>(P.q + static_cast<int64_t>(r) * P.q_stride) : reinterpret_cast<const char*>(P.q_logits + static_cast<int64_t>(r) * P.q_logits_stride);
  const bool q_vec = ((reinterpret_cast<uintptr_t>(q_row) - static_cast<uintptr_t>(off) * (Q == 1 ? 4 : 2)) & 15u) == 0u;
  if (tid == 0) {
    VerifyRow& x = s.row;
    x.z_row = z_row; x.q_row = q_row; x.off = off; x.V = V;
    x.cut = P.tau != nullptr; x.tau = P.tau ? P.tau[row] : -INFINITY; x.c2 = Q != 0 ? exp2_scale(P.temperature) : 0.0f;
  }
  auto whole = [&](int c) { const int base = 8 * c - off; return base >= 0 && base + 8 <= V; };
  constexpr uint32_t kOut = F32 ? 0xFF800000u : 0xFF80u;
  if (z_cached) {
#pragma unroll 1
    for (int c = w0 + lane; c < w1; c += 32) {
      if (whole(c)) {
        const char* src = z_row + static_cast<int64_t>(8 * c - off) * kSize;
        cp_async16(zs + c, src);
        if (F32) cp_async16(zs + per + c, src + 16);
      } else {
        zs[c] = verify_far<F32>(z_row, off, V, c, 0, false, kOut);
        if (F32) zs[per + c] = verify_far<F32>(z_row, off, V, c, 1, false, kOut);
      }
    }
  }
  cp_async_commit();
  if (Q != 0 && has_q && q_cached) {
#pragma unroll 1
    for (int c = w0 + lane; c < w1; c += 32) {
      if (q_vec && whole(c)) {
        const char* src = q_row + static_cast<int64_t>(8 * c - off) * (Q == 1 ? 4 : 2);
        cp_async16(qs + c, src);
        if (Q == 1) cp_async16(qs + per + c, src + 16);
      } else {
        qs[c] = verify_far<Q == 1>(q_row, off, V, c, 0, false, Q == 1 ? 0u : 0xFF80u);
        if (Q == 1) qs[per + c] = verify_far<Q == 1>(q_row, off, V, c, 1, false, 0u);
      }
    }
  }
  cp_async_commit();
  // The scalars of the accept test go out under the copies. They are the last warp's, which has the fewest chunks.
  const float c2 = Q != 0 ? exp2_scale(P.temperature) : 0.0f;
  const bool tester = Q != 0 && warp == kVerifyWarps - 1;
  const float u_final = Q != 0 && P.u_final ? P.u_final[0] : 0.0f;           // (wanted at the very end)
  const bool tests = tester && has_q && (lane & 15) == 0, drafter = lane >= 16;
  VerifyTest<F32, Q> t;
  t.load(P, rd, tests, false, r);
  // half h of a chunk as it lies in memory (BF16: the whole chunk, whichever half)
  auto z_raw = [&](int c, int h) { return z_cached ? zs[(F32 && h ? per : 0) + c] : verify_far<F32>(z_row, off, V, c, h, true, kOut); };
  bool joined = C == 1;                                                     // every block of the cluster runs: its shared memory may be written to
  auto join = [&]() { if (!joined) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); joined = true; };
  // a warp's value to every block of the cluster (or to block 0 alone)
  auto push = [&](unsigned long long* slots, uint64_t v, bool all) { if (lane < (all ? C : 1)) cst_u64(cluster_addr(&slots[rank], lane), v); };

  // ---- the row's maximum (greedy: with its lowest index) ------------------------------------------------------------------------------
  float vmax = 0.0f;
  cp_async_wait<1>();                                                       // (a thread reads back its own chunks: no barrier)
  if (given_max) { vmax = canon_zero(P.row_max[row]); __syncthreads(); }
  else {
    // Per half its maximum alone. NaN follows the packed order (a positive NaN above +inf, a negative one below -inf): a half that holds one is compared
    // element by element. Greedy looks for the index once, at the end.
    float top = -INFINITY;
    int top_c = w0 + lane < w1 ? 2 * (w0 + lane) : -1;
    uint64_t best = 0ull;
    auto elements = [&](int ch, bool any, float value) {                    // those of half ch & 1 of chunk ch >> 1 that are in the row and (any or they equal value)
      const uint4 v = z_raw(ch >> 1, ch & 1);
      float2 z[2];
      verify_pairs<F32>(v, ch & 1, z);
#pragma unroll 1
      for (int e = 0; e < 4; e++) {
        const float2 z2 = (e & 2) ? z[1] : z[0];
        const float ze = (e & 1) ? z2.y : z2.x;
        const int i = 4 * ch + e - off;
        if (i < 0 || i >= V || !(any || ze == value)) continue;
        const uint64_t p = pack_best(ze, static_cast<uint32_t>(i));
        best = p > best ? p : best;
      }
    };
#pragma unroll 1
    for (int c = w0 + lane; c < w1; c += 32) {
      uint4 v = z_raw(c, 0);
#pragma unroll 1
      for (int h = 0; h < 2; h++) {
        float mx;
        if (F32) {
          if (h) v = z_raw(c, 1);
          asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(__uint_as_float(v.x)), "f"(__uint_as_float(v.y)));
          asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(mx), "f"(__uint_as_float(v.z)));
          asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(mx), "f"(__uint_as_float(v.w)));
        } else {
          const uint32_t a = h ? v.z : v.x, b = h ? v.w : v.y;
          const __nv_bfloat162 m = __hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
          const float l = __low2float(m), u = __high2float(m);
          asm("max.NaN.f32 %0, %1, %2;" : "=f"(mx) : "f"(l), "f"(u));
        }
        if (mx > top) { top = mx; top_c = 2 * c + h; }
        if (mx != mx) elements(2 * c + h, true, 0.0f);
      }
    }
    if (Q == 0 && top_c >= 0) {
      // (a row of nothing but -inf: this thread's first element that is in the row)
      elements(top_c, false, canon_zero(top));
      if (best == 0ull) elements(top_c + 1, false, canon_zero(top));
    }
    best = Q != 0 ? static_cast<uint64_t>(warp_max_u32(max(fkey(canon_zero(top)), static_cast<uint32_t>(best >> 32)))) : warp_max_u64(best);   // (stochastic: the value alone)
    if (lane == 0) s.best[warp] = best;
    __syncthreads();
    join();
    if (warp == 0) push(s.x_best, warp_max_u64(lane < kVerifyWarps ? s.best[lane] : 0ull), Q != 0);
    cluster_sync(C);
    if (Q == 0) {
      if (rank == 0 && warp == 0) {
        const int pick = static_cast<int>(best_index(warp_max_u64(lane < C ? s.x_best[lane] : 0ull)));
        verify_arrive(P, rd, r, launch, r < L && pick != verify_draft(P, rd, r), pick);
      }
      return;
    }
    vmax = fkey_inv(warp_max_u32(lane < C ? static_cast<uint32_t>(s.x_best[lane]) : 0u));
  }
  if (Q == 0) return;

  // ---- the kept set's mass and the accept test ---------------------------------------------------------------------------------------------
  const bool keep_w = !kStats && !(kGumbel && !has_q);                      // the weights replace the logits
  // a chunk's weights, as floors, from its logits in shared memory; nothing kept of it costs its maximum
  auto weigh = [&](int c, FloorSum& sum, float2 (&w)[4]) {
    const float tau = s.row.tau;
    float2 z[4];
    const uint4 v = zs[c];
    if (F32) {
      const uint4 b = zs[per + c];
      z[0] = make_float2(__uint_as_float(v.x), __uint_as_float(v.y)); z[1] = make_float2(__uint_as_float(v.z), __uint_as_float(v.w));
      z[2] = make_float2(__uint_as_float(b.x), __uint_as_float(b.y)); z[3] = make_float2(__uint_as_float(b.z), __uint_as_float(b.w));
    } else {
      z[0] = make_float2(bf16_lo(v.x), bf16_hi(v.x)); z[1] = make_float2(bf16_lo(v.y), bf16_hi(v.y));
      z[2] = make_float2(bf16_lo(v.z), bf16_hi(v.z)); z[3] = make_float2(bf16_lo(v.w), bf16_hi(v.w));
    }
    const bool none = s.row.cut && !(fmaxf(fmaxf(fmaxf(z[0].x, z[0].y), fmaxf(z[1].x, z[1].y)), fmaxf(fmaxf(z[2].x, z[2].y), fmaxf(z[3].x, z[3].y))) >= tau);
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = make_float2(0.0f, 0.0f);
    if (!none) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        z[k] = __fadd2_rn(z[k], make_float2(0.0f, 0.0f));
        const float2 x = weight_f2(z[k].x, z[k].y, vmax, c2);
        w[k] = sum.add(make_float2(z[k].x >= tau ? x.x : 0.0f, z[k].y >= tau ? x.y : 0.0f));
      }
    }
    if (keep_w) {
      zs[c] = make_uint4(__float_as_uint(w[0].x), __float_as_uint(w[0].y), __float_as_uint(w[1].x), __float_as_uint(w[1].y));
      zs[per + c] = make_uint4(__float_as_uint(w[2].x), __float_as_uint(w[2].y), __float_as_uint(w[3].x), __float_as_uint(w[3].y));
    }
  };
  bool residual = false;
  auto half_weight = [&](int c, int h) {                                    // (of the weights that replaced the logits)
    const uint4 v = zs[(h ? per : 0) + c];
    const float4 w = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
    if (!residual) return w;
    const uint4 qr = q_cached ? qs[(Q == 1 && h ? per : 0) + c] : verify_far<Q == 1>(q_row, off, V, c, h, q_vec, Q == 1 ? 0u : 0xFF80u);
    return verify_rest<F32, Q>(s.row, w, qr, c, h, vmax);
  };
  unsigned long long mass;
  VerifySums shares;                                                        // the blocks' shares of what is drawn from
  {
    uint64_t own = 0ull;
#pragma unroll 1
    for (int c = w0 + lane; c < w1; c += 32) {
      if (z_cached) {
        FloorSum sum;
        float2 w[4];
        weigh(c, sum, w);
        const uint64_t sum_c = sum.sum();
        own += sum_c;
        if (!kStats) sums[c] = sum_c;
      } else {
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
          const float4 x = verify_weights<F32>(s.row, z_raw(c, h), h, vmax);
          FloorSum sum;
          sum.add(make_float2(x.x, x.y)); sum.add(make_float2(x.z, x.w));
          own += sum.sum();
        }
      }
    }
    float t_q = 0.0f;
    if (Q == 2 && tests && drafter) { s.row.qv = t.vmax; s.row.q_of.init(t.mass); t_q = t.prob(t.vmax, t.mass, c2); }   // (the drafter's side, before the mass is known)
    own = warp_sum_u64(own);
    if (lane == 0) s.own[warp] = own;
    __syncthreads();
    join();
    if (warp == 0) {
      const uint64_t block = warp_sum_u64(lane < kVerifyWarps ? s.own[lane] : 0ull);
      push(s.x_own, block, true);
      if (lane == 0) s.own_block = block;
    }
    cluster_sync(C);
    mass = verify_sums(s.x_own, C, shares);
    if (kStats) {
      if (rank == 0 && tid == 0) { P.ws->vmax[row] = vmax; P.ws->mass[row] = mass; }
      return;
    }
    if (has_q) {
      if (tester) {
        const float pq = drafter ? t_q : t.prob(vmax, mass, c2);
        const bool no = t.rejects(pq);
        if (lane == 0) {
          if (rank == 0 && P.out_p_draft) P.out_p_draft[r] = pq;
          s.reject = no; s.row.p_of.init(mass);
        }
      }
      __syncthreads();
      if (!s.reject) {
        if (rank == 0 && warp == 0) verify_arrive(P, rd, r, launch, false, -1);
        cp_async_wait<0>();
        return;
      }
    }
  }

  // ---- the draw: over the residual max(p - q, 0) of a rejected draft, over p itself on the bonus row or where the residual is empty -----------
  cp_async_wait<0>();
  auto deliver = [&](int token) { verify_arrive(P, rd, r, launch, r < L, token); };   // one whole warp of the cluster
  // The sums of the draw: the residual's, and where that is empty the row's own once more (the mass's sums will do where there is no draft). Or, in the reference's
  // form (kernels/common/sample.metal:322-346), the best of ln(p - q) + noise of stream 4000, and where nothing is left the best of the row's own Gumbel keys.
  const unsigned long long* parts = reinterpret_cast<const unsigned long long*>(s.own);
  uint64_t there = mass;                                                    // the weight of all blocks (or the best key)
  if (has_q || kGumbel) {
    parts = reinterpret_cast<const unsigned long long*>(s.res);
    residual = has_q;
    bool first = true;
#pragma unroll 1
    for (;; residual = first = false) {
      uint64_t w = 0ull;
      if (mass > 0ull && !(kGumbel && !residual)) {
#pragma unroll 1
        for (int c = w0 + lane; c < w1; c += 32) {
          uint64_t v = 0ull;
          if (first) {
            float2 x[4];
            FloorSum sum;
            {
              const uint4 a = zs[c], b = zs[per + c];
              x[0] = make_float2(__uint_as_float(a.x), __uint_as_float(a.y)); x[1] = make_float2(__uint_as_float(a.z), __uint_as_float(a.w));
              x[2] = make_float2(__uint_as_float(b.x), __uint_as_float(b.y)); x[3] = make_float2(__uint_as_float(b.z), __uint_as_float(b.w));
            }
            {
              uint32_t any = 0u;
              bool below = false;
#pragma unroll
              for (int k = 0; k < 4; k++) any |= __float_as_uint(x[k].x) | __float_as_uint(x[k].y);
              if (any || Q == 1) {
                float2 q[4];
                uint4 a, b;
                if (q_cached) { a = qs[c]; if (Q == 1) b = qs[per + c]; }
                else { a = verify_far<Q == 1>(q_row, off, V, c, 0, q_vec, Q == 1 ? 0u : 0xFF80u); if (Q == 1) b = verify_far<Q == 1>(q_row, off, V, c, 1, q_vec, 0u); }
                if (Q == 1) {
                  q[0] = make_float2(__uint_as_float(a.x), __uint_as_float(a.y)); q[1] = make_float2(__uint_as_float(a.z), __uint_as_float(a.w));
                  q[2] = make_float2(__uint_as_float(b.x), __uint_as_float(b.y)); q[3] = make_float2(__uint_as_float(b.z), __uint_as_float(b.w));
                  below = fminf(fminf(fminf(q[0].x, q[0].y), fminf(q[1].x, q[1].y)), fminf(fminf(q[2].x, q[2].y), fminf(q[3].x, q[3].y))) < 0.0f;
                } else {
                  const ProbScale q_of = s.row.q_of;
                  const float qv = s.row.qv;
                  const uint32_t u[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                  for (int k = 0; k < 4; k++) {
                    const float2 z = __fadd2_rn(make_float2(bf16_lo(u[k]), bf16_hi(u[k])), make_float2(0.0f, 0.0f));
                    uint2 t, l;
                    q[k] = q_of.of(floor2(weight_f2(z.x, z.y, qv, c2), t, l));
                  }
                }
                const ProbScale p_of = s.row.p_of;
                if (below) {
                  const float4 l = verify_below_zero<F32>(s.row, c, 0, vmax), u = verify_below_zero<F32>(s.row, c, 1, vmax);
                  x[0] = make_float2(l.x, l.y); x[1] = make_float2(l.z, l.w); x[2] = make_float2(u.x, u.y); x[3] = make_float2(u.z, u.w);
                  v += verify_wide(l, u);
                } else if (any)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                  const float2 d = __fadd2_rn(p_of.of(x[k]), make_float2(-q[k].x, -q[k].y));
                  x[k] = __fmul2_rn(make_float2(x[k].x > 0.0f ? fmaxf(d.x, 0.0f) : 0.0f, x[k].y > 0.0f ? fmaxf(d.y, 0.0f) : 0.0f), make_float2(1099511627776.0f, 1099511627776.0f));
                  sum.add(x[k]);
                }
              }
            }
            if (kGumbel || q_cached) {
              uint4* to = kGumbel ? zs : qs;
              to[c] = make_uint4(__float_as_uint(x[0].x), __float_as_uint(x[0].y), __float_as_uint(x[1].x), __float_as_uint(x[1].y));
              to[per + c] = make_uint4(__float_as_uint(x[2].x), __float_as_uint(x[2].y), __float_as_uint(x[3].x), __float_as_uint(x[3].y));
            }
            v += sum.sum();
          } else {
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
              const float4 y = half_weight(c, h);
              FloorSum sum;
              sum.add(make_float2(y.x, y.y)); sum.add(make_float2(y.z, y.w));
              v += sum.sum();
            }
          }
          sums[c] = v;
          w += v;
        }
      }
      w = warp_sum_u64(w);
      if (kGumbel) w = mass == 0ull ? 0ull : verify_best_key<F32>(P, rd, s, zs, w0, w1, per, row, residual, has_q, residual ? w : 0ull, vmax);
      if (lane == 0) s.res[warp] = w;
      __syncthreads();
      if (warp == 0) {
        w = lane < kVerifyWarps ? s.res[lane] : 0ull;
        push(s.x_res, kGumbel ? warp_max_u64(w) : warp_sum_u64(w), true);
      }
      cluster_sync(C);
      there = kGumbel ? warp_max_u64(lane < C ? s.x_res[lane] : 0ull) : verify_sums(s.x_res, C, shares);
      if (there || !residual) break;
      cluster_sync(C);                                                      // (everybody has read the slots)
    }
  }
  if (kGumbel) {
    if (rank == 0 && warp == 0) deliver(there ? static_cast<int>(best_index(there)) : -1);
    return;
  }
  uint64_t left = cdf_target(P.u_final ? u_final : uniform01(rd.seed, rd.step, 4000u, 0u), residual ? there : mass);
  const int block = verify_slot(shares, left);
  if (block != rank) {                                                      // none: a row with no weight at all (empty or all -inf), or a given mass that is not the row's
    if (block < 0 && rank == 0 && warp == 0) deliver(-1);
    return;
  }
  VerifySums mine;
  verify_sums(parts, kVerifyWarps, mine);
  const int part = verify_slot(mine, left);
  if (warp != max(part, 0)) return;
  // the first element, in index order, at which the running weight passes the target: the chunk from the chunks' sums, then a lane for each of its elements
  // ... where the draw's weights lie: in the drafter's place, or where the row itself is drawn from in the logits' place; a residual that was not kept is formed again
  const bool kept_values = q_cached && residual;
  int token = -1;
#pragma unroll 1
  for (int b0 = w0; b0 < w1 && part >= 0; b0 += 32) {
    const int c = b0 + lane;
    uint64_t sum = 0ull;
    if (c < w1) sum = sums[c];
    uint64_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
    uint64_t run = incl - sum;
    const uint32_t hit = __ballot_sync(kFull, run <= left && left < incl);
    if (hit) {
      const int ch = b0 + __ffs(static_cast<int>(hit)) - 1, e = lane & 7, h = e >> 2;
      run = __shfl_sync(kFull, run, ch - b0);
      uint64_t v;
      if (kept_values || !residual) v = __float2ull_rz(reinterpret_cast<const float*>((kept_values ? qs : zs) + (h ? per : 0) + ch)[e & 3]);
      else {
        const float4 x = half_weight(ch, h);
        v = __float2ull_rz((e & 2) ? ((e & 1) ? x.w : x.z) : ((e & 1) ? x.y : x.x));
      }
      uint64_t upto = v;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, upto, o); if (e >= o) upto += t; }
      const uint32_t at = __ballot_sync(kFull, run + upto - v <= left && left < run + upto) & 0xFFu;
      if (at) token = 8 * ch + __ffs(static_cast<int>(at)) - 1 - off;
      break;
    }
    left -= __shfl_sync(kFull, incl, 31);
  }
  deliver(token);
}

template <bool F32, int Q, int kMode>
static __global__ void __launch_bounds__(kVerifyThreads, 2) verify_kernel(const __grid_constant__ VerifyDev P, int C, int z_cached, int q_cached) {
  extern __shared__ __align__(16) uint4 v_smem[];
  __shared__ VerifySmem s;
  const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0, r = static_cast<int>(blockIdx.x) / C;
  after_predecessor();
  unsigned long long launch;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(launch) : "l"(&P.ws->launches) : "memory");
  VerifyRound rd;
  if (verify_begin(P, rd, kMode != kVerifyStats) && r <= rd.L) {                                   // (a state may verify fewer rows than the launch has clusters)
    if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this block runs, and has read the state
    verify_row<F32, Q, kMode>(P, rd, r, rank, C, launch, z_cached != 0, q_cached != 0, v_smem, s);
  }
}

}  // namespace lm

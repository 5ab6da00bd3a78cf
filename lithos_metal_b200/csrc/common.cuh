// Device helpers shared by the generation-control kernels (sm_100a).
//
// Everything that feeds an integer decision (token ids, kept sets, accept counts) is written with explicit
// round-to-nearest intrinsics so that the compiler cannot contract or reorder it: the same sequence of IEEE
// operations on a CPU gives the same bits.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/lithos_b200.h"

namespace lm {

#ifndef LM_BLOCK
#define LM_BLOCK 1024
#endif
constexpr int kBlock = LM_BLOCK;       // threads per block of the row kernels
constexpr int kWarps = kBlock / 32;
constexpr int kChunk = 8;              // consecutive logits one thread takes per step (one 128-bit load of BF16)
constexpr uint32_t kFull = 0xFFFFFFFFu;

// A kernel that may be launched beside its predecessor in the stream (launch_beside, host.cuh): here that one is complete and what it wrote is
// visible. Every thread calls this before it touches device memory, and before it returns. What is launched behind this kernel the same way may
// then be made ready (its blocks wait here in turn).
__device__ __forceinline__ void after_predecessor() { asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory"); }

// ---- element access ----------------------------------------------------------------------------------------

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// A bit per logit of a chunk from the masks of packed compares.
__device__ __forceinline__ uint32_t mask8(uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  return (m0 & 1u) | ((m0 >> 15) & 2u) | ((m1 & 1u) << 2) | ((m1 >> 13) & 8u) | ((m2 & 1u) << 4) | ((m2 >> 11) & 32u) | ((m3 & 1u) << 6) | ((m3 >> 9) & 128u);
}
// 8-bit mask of the logits of a chunk of BF16 codes that are at or above the code in both halves of tau_code2.
__device__ __forceinline__ uint32_t kept_mask8(const uint4 q, uint32_t tau_code2) {
  const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&tau_code2);
  const uint32_t m0 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.x), t2), m1 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.y), t2);
  const uint32_t m2 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.z), t2), m3 = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.w), t2);
  return (m0 | m1 | m2 | m3) == 0u ? 0u : mask8(m0, m1, m2, m3);
}
// The same logits in no particular order: bits 0..3 and 16..19, one per logit (where they are only counted).
__device__ __forceinline__ uint32_t kept_bits8(const uint4 q, uint32_t tau_code2) {
  const __nv_bfloat162 t2 = *reinterpret_cast<const __nv_bfloat162*>(&tau_code2);
  return (__hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.x), t2) & 0x00010001u) | (__hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.y), t2) & 0x00020002u) |
         (__hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.z), t2) & 0x00040004u) | (__hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&q.w), t2) & 0x00080008u);
}

// Monotone 32-bit key of a float: a > b  <=>  fkey(a) > fkey(b) (for non-NaN, with -0 canonicalised to +0 first).
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
__device__ __forceinline__ float canon_zero(float z) { return z == 0.0f ? 0.0f : z; }

// Repetition then presence penalty on one widened logit (both binary32, round to nearest).
__device__ __forceinline__ float penalise(float z, float rho, float pi) {
  z = (z > 0.0f) ? __fdiv_rn(z, rho) : __fmul_rn(z, rho);
  return __fsub_rn(z, pi);
}

// One row of logits as the kernels see it: widened to float, penalties applied on the fly from a bitmap of the
// row's distinct history ids (shared memory), -0 folded into +0.
struct RowView {
  const void* row;
  int dtype;
  int vocab;
  bool aligned;            // row start is 16-byte aligned: 128-bit loads are legal
  const uint32_t* pen;     // bitmap over [0, vocab) or nullptr
  float rho, pi;
};

// Elements [8c, 8c + 8) of the row; returns how many of them exist (0..8).
__device__ __forceinline__ int load_chunk(const RowView& rv, int c, float z[kChunk]) {
  const int base = c * kChunk;
  const int n = min(kChunk, rv.vocab - base);
  if (n <= 0) return 0;
  if (rv.dtype == LM_DTYPE_BF16) {
    const uint16_t* p = reinterpret_cast<const uint16_t*>(rv.row) + base;
    if (n == kChunk && rv.aligned) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
      z[0] = bf16_lo(q.x); z[1] = bf16_hi(q.x); z[2] = bf16_lo(q.y); z[3] = bf16_hi(q.y);
      z[4] = bf16_lo(q.z); z[5] = bf16_hi(q.z); z[6] = bf16_lo(q.w); z[7] = bf16_hi(q.w);
    } else {
#pragma unroll
      for (int e = 0; e < kChunk; e++) z[e] = (e < n) ? __uint_as_float(static_cast<uint32_t>(__ldg(p + e)) << 16) : 0.0f;
    }
  } else {
    const float* p = reinterpret_cast<const float*>(rv.row) + base;
    if (n == kChunk && rv.aligned) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
      z[0] = a.x; z[1] = a.y; z[2] = a.z; z[3] = a.w; z[4] = b.x; z[5] = b.y; z[6] = b.z; z[7] = b.w;
    } else {
#pragma unroll
      for (int e = 0; e < kChunk; e++) z[e] = (e < n) ? __ldg(p + e) : 0.0f;
    }
  }
  if (rv.pen != nullptr) {
    const uint32_t bits = (rv.pen[c >> 2] >> ((c & 3) * 8)) & 0xFFu;
    if (bits) {
#pragma unroll
      for (int e = 0; e < kChunk; e++) if ((bits >> e) & 1u) z[e] = penalise(z[e], rv.rho, rv.pi);
    }
  }
#pragma unroll
  for (int e = 0; e < kChunk; e++) z[e] = canon_zero(z[e]);
  return n;
}

// ---- the counter-based noise of the reference's draw --------------------------------------------------------

__host__ __device__ __forceinline__ float uniform01(uint64_t seed, uint32_t step, uint32_t t, uint32_t i) {
  uint64_t x = seed + static_cast<uint64_t>(step) * 0x9E3779B97F4A7C15ull + static_cast<uint64_t>(t) * 0xC2B2AE3D27D4EB4Full +
               static_cast<uint64_t>(i) * 0x165667B19E3779F9ull;
  x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull; x ^= x >> 27; x *= 0x94D049BB133111EBull; x ^= x >> 31;
  return (static_cast<float>((x >> 41) & 0x7FFFFFull) + 0.5f) * (1.0f / 8388608.0f);
}
__device__ __forceinline__ float gumbel(uint64_t seed, uint32_t step, uint32_t t, uint32_t i) {
  return -logf(-logf(uniform01(seed, step, t, i)));
}

// ---- the integer-exact weights of the inverse-CDF draw ------------------------------------------------------

// 2^x for x <= 0: round-to-nearest split, degree-5 polynomial with fused multiply-adds, exact power-of-two scaling.
__device__ __forceinline__ float spec_exp2(float x) {
  if (!(x > -100.0f)) return 0.0f;
  x = fminf(x, 0.0f);
  const float n = rintf(x);
  const float f = __fsub_rn(x, n);
  float p = 0x1.5bba20p-10f;
  p = __fmaf_rn(p, f, 0x1.3cea88p-7f);
  p = __fmaf_rn(p, f, 0x1.c6b752p-5f);
  p = __fmaf_rn(p, f, 0x1.ebf9bcp-3f);
  p = __fmaf_rn(p, f, 0x1.62e42ap-1f);
  p = __fmaf_rn(p, f, 1.0f);
  return __fmul_rn(p, __int_as_float((static_cast<int>(n) + 127) << 23));
}
// log2(e) / T as a binary32: divided in binary64, rounded once.
__device__ __forceinline__ float exp2_scale(float temperature) {
  return __double2float_rn(__ddiv_rn(1.4426950408889634, static_cast<double>(temperature)));
}
// floor(2^40 * spec_exp2(fl32(fl32(z - vmax) * c)))
__device__ __forceinline__ uint64_t weight_q40(float z, float vmax, float c) {
  const float x = __fmul_rn(__fsub_rn(z, vmax), c);
  return __float2ull_rz(__fmul_rn(spec_exp2(x), 1099511627776.0f));
}
// Two weights at once on the packed binary32 instructions of sm_100 (fma.rn.f32x2 and friends): element for element the
// operations of weight_q40 up to its conversion, so the same bits: a weight is the floor of what this returns. (z - vmax is formed as z + (-vmax); the two
// exact power-of-two scalings, by 2^n and by 2^40, are one multiplication by 2^(n + 40).)
__device__ __forceinline__ float2 weight_f2(float z0, float z1, float vmax, float c) {
  const float2 x = __fmul2_rn(__fadd2_rn(make_float2(z0, z1), make_float2(-vmax, -vmax)), make_float2(c, c));
  const float x0 = fminf(fmaxf(x.x, -100.0f), 0.0f), x1 = fminf(fmaxf(x.y, -100.0f), 0.0f);   // (at -100 and below, and for a NaN, 2^-60: floor 0, as spec_exp2 has it)
  // round to nearest (ties to even) by adding and subtracting 1.5 * 2^23: for -100 < x <= 0 the sum has an ulp of 1, so this is
  // rintf(x) exactly, and the integer sits in the low bits of the sum (no conversion instructions, which run at a quarter of the rate)
  const float kMagic = 12582912.0f;
  const float2 t = __fadd2_rn(make_float2(x0, x1), make_float2(kMagic, kMagic));
  const float2 n = __fadd2_rn(t, make_float2(-kMagic, -kMagic));
  const float2 f = __fadd2_rn(make_float2(x0, x1), make_float2(-n.x, -n.y));
  float2 p = make_float2(0x1.5bba20p-10f, 0x1.5bba20p-10f);
  p = __ffma2_rn(p, f, make_float2(0x1.3cea88p-7f, 0x1.3cea88p-7f));
  p = __ffma2_rn(p, f, make_float2(0x1.c6b752p-5f, 0x1.c6b752p-5f));
  p = __ffma2_rn(p, f, make_float2(0x1.ebf9bcp-3f, 0x1.ebf9bcp-3f));
  p = __ffma2_rn(p, f, make_float2(0x1.62e42ap-1f, 0x1.62e42ap-1f));
  p = __ffma2_rn(p, f, make_float2(1.0f, 1.0f));
  // (t's bits are 0x4B400000 + n: shifted by 23, the constant is gone and n + 167 is an exponent)
  return __fmul2_rn(p, make_float2(__int_as_float((__float_as_int(t.x) << 23) + (167 << 23)), __int_as_float((__float_as_int(t.y) << 23) + (167 << 23))));
}
__device__ __forceinline__ void weight_q40_x2(float z0, float z1, float vmax, float c, uint64_t& w0, uint64_t& w1) {
  const float2 r = weight_f2(z0, z1, vmax, c);
  w0 = __float2ull_rz(r.x); w1 = __float2ull_rz(r.y);
}
// The floors of two binary32 x, 0 <= x <= 2^40, without the conversion to 64 bits (which runs at an eighth of the rate): 2^-17 x and what is left of x are
// rounded down against 2^23, so that the integers lie in the sums' low bits. `top`, `low`: their bit patterns, each less 0x4B000000 an integer; floor =
// top << 17 | low. Returned: the floors as binary32 where they fit 24 bits (they do for a weight: one below 2^24 is an integer below that, a larger one is x).
__device__ __forceinline__ float2 floor2(float2 x, uint2& top, uint2& low) {
  const float2 t = __fadd2_rd(__fmul2_rn(x, make_float2(0x1p-17f, 0x1p-17f)), make_float2(8388608.0f, 8388608.0f));
  const float2 h = __fadd2_rn(t, make_float2(-8388608.0f, -8388608.0f));
  const float2 u = __fadd2_rd(__ffma2_rn(h, make_float2(-131072.0f, -131072.0f), x), make_float2(8388608.0f, 8388608.0f));
  top = make_uint2(__float_as_uint(t.x), __float_as_uint(t.y)); low = make_uint2(__float_as_uint(u.x), __float_as_uint(u.y));
  return __ffma2_rn(h, make_float2(131072.0f, 131072.0f), __fadd2_rn(u, make_float2(-8388608.0f, -8388608.0f)));
}
// A sum of such floors, eight at most at a time (2^26 and 2^20 in all).
struct FloorSum {
  uint32_t top = 0u, low = 0u, n = 0u;
  __device__ __forceinline__ float2 add(float2 x) {
    uint2 t, l;
    const float2 w = floor2(x, t, l);
    top += t.x + t.y; low += l.x + l.y; n += 2u;
    return w;
  }
  __device__ __forceinline__ bool beyond() const { return top - n * 0x4B000000u > 8388608u; }   // more than 2^40 in all, or an x above 2^40 (2^64 at most) among them: no sum
  __device__ __forceinline__ uint64_t sum() const { return (static_cast<uint64_t>(top - n * 0x4B000000u) << 17) + (low - n * 0x4B000000u); }
};
// floor(floor(u * 2^24) * total / 2^24), u clamped to [0, 1 - 2^-24]
__device__ __forceinline__ uint64_t cdf_target(float u, uint64_t total) {
  long long u24 = (u > 0.0f) ? __float2ll_rz(__fmul_rn(u, 16777216.0f)) : 0ll;
  if (u24 > 16777215ll) u24 = 16777215ll;
  const uint64_t a = static_cast<uint64_t>(u24);
  return (__umul64hi(total, a) << 40) | ((total * a) >> 24);
}
// binary32 probability of one token: fl32(double(w) / double(k))
__device__ __forceinline__ float prob_q40(uint64_t w, uint64_t k) {
  return __double2float_rn(__ddiv_rn(__ull2double_rn(w), __ull2double_rn(k)));
}
// fixed-point residual weight floor(2^40 * r) for a positive binary32 r <= 1
__device__ __forceinline__ uint64_t residual_q40(float r) { return __float2ull_rz(__fmul_rn(r, 1099511627776.0f)); }

// ---- block-wide reductions over kBlock threads (scratch: 32 entries of the type in shared memory) --------------

// 32-bit warp reductions by butterfly shuffles. (The single-instruction warp reduction, redux.sync, measured about 0.3 us per
// use on B200 when every warp of a block issues it: far slower than five shuffles.)
__device__ __forceinline__ uint32_t warp_sum_u32(uint32_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ uint32_t warp_max_u32(uint32_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ uint32_t warp_min_u32(uint32_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ uint64_t warp_max_u64(uint64_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) { const uint64_t t = __shfl_xor_sync(kFull, v, o); v = t > v ? t : v; }
  return v;
}
__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// All threads of the block must call; every thread gets the result. `scratch` holds blockDim.x/32 entries.
__device__ __forceinline__ uint64_t block_max_u64(uint64_t v, uint64_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_max_u64(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  uint64_t r = (lane < nw) ? scratch[lane] : 0ull;
  return warp_max_u64(r);
}
__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v, uint64_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum_u64(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  uint64_t r = (lane < nw) ? scratch[lane] : 0ull;
  return warp_sum_u64(r);
}
__device__ __forceinline__ double block_sum_f64(double v, uint64_t* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* s = reinterpret_cast<double*>(scratch);
  v = warp_sum_f64(v);
  __syncthreads();
  if (lane == 0) s[warp] = v;
  __syncthreads();
  double r = (lane < nw) ? s[lane] : 0.0;
  return warp_sum_f64(r);
}
// Exclusive prefix sum over the block's threads in thread order; *total gets the block sum.
__device__ __forceinline__ uint64_t block_exclusive_scan_u64(uint64_t v, uint64_t* scratch, uint64_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint64_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, incl, o); if (lane >= o) incl += t; }
  __syncthreads();
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  uint64_t w = (lane < nw) ? scratch[lane] : 0ull;
  uint64_t winc = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint64_t t = __shfl_up_sync(kFull, winc, o); if (lane >= o) winc += t; }
  const uint64_t warp_base = __shfl_sync(kFull, winc - w, warp);
  if (total) *total = __shfl_sync(kFull, winc, nw - 1);
  return warp_base + incl - v;
}

// A row's token, 32 or 64 bits wide.
__device__ __forceinline__ void store_token(int32_t* out, uint32_t flags, int row, int token) {
  if (flags & LM_FLAG_TOKENS_I64) reinterpret_cast<int64_t*>(out)[row] = token; else out[row] = token;
}

// Packed (value, index) for argmax with ties -> lowest index: larger packed value wins.
__device__ __forceinline__ uint64_t pack_best(float v, uint32_t idx) { return (static_cast<uint64_t>(fkey(v)) << 32) | (0xFFFFFFFFu - idx); }
__device__ __forceinline__ uint32_t best_index(uint64_t p) { return 0xFFFFFFFFu - static_cast<uint32_t>(p); }
__device__ __forceinline__ float best_value(uint64_t p) { return fkey_inv(static_cast<uint32_t>(p >> 32)); }

// ---- exp(y) for y <= 0 in FP64: the table-driven exponential (P. T. P. Tang, ACM TOMS 15(2), 1989) -----------------------------
// y = (64 m + j) ln2 / 64 + r, |r| <= ln2 / 128; exp(y) = 2^m 2^(j/64) e^r, e^r by its Taylor polynomial of degree 5 (remainder
// r^6 / 720 <= 3.6e-17), the reduction in two parts so that r carries no more than its own rounding. Below -690: 0.
__device__ __forceinline__ double exp64(double y, const double* tab) {
  if (!(y > -690.0)) return 0.0;
  const double t = __fma_rn(y, 0x1.71547652b82fep+6, 0x1.8p52);            // 64 / ln2; the integer sits in the low bits
  const int n = __double2loint(t);
  const double k = __dadd_rn(t, -0x1.8p52);
  double r = __fma_rn(k, -0x1.62e42fef00000p-7, y);                        // ln2 / 64, its first 33 bits ...
  r = __fma_rn(k, -0x1.473de6af278edp-40, r);                              // ... and the rest
  double p = __fma_rn(r, 1.0 / 120.0, 1.0 / 24.0);
  p = __fma_rn(p, r, 1.0 / 6.0);
  p = __fma_rn(p, r, 0.5);
  p = __fma_rn(p, r, 1.0);
  p = __fma_rn(p, r, 1.0);
  p = __dmul_rn(p, tab[n & 63]);
  return __hiloint2double(__double2hiint(p) + ((n >> 6) << 20), __double2loint(p));
}

__device__ __forceinline__ float ex2_approx(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// A row's softmass in FP32 is a sum of 2^(z c + nb), c = log2(e) / T, nb = fl32(-vmax c). The rounding of nb is a factor common to all terms and
// is taken out afterwards -- as long as it is a fraction of a binade. At |vmax| / T of 2^20 it is 2^-4 at most; where |vmax| / T reaches 2^29 or so
// it is 2^5 binades and more, and the largest term may overflow (or all of them vanish). Beyond this line the sum is formed in FP64.
constexpr double kMassExponent = 0x1p20;

// ---- Gumbel keys, the two logarithms only where they can matter --------------------------------------------------------------------
// key = z / T + g, g = -ln(-ln u), u = (h + 1/2) / 2^23 from 23 bits of the hash. key >= B needs -ln u <= exp(z / T - B), and 1 - u <=
// -ln u: a logit with (2^23 - h) > 2^23 exp(z / T - B) + 1 cannot reach B. One hash and one ex2 per logit decide that; the few that pass
// get the exact key. B is a key already seen, less the 4e-6 of the near-tie flag and the rounding of the test itself (kSlack).
constexpr uint64_t kHashStep = 0x165667B19E3779F9ull;   // (uniform01: what one index adds)
struct GumbelScan {
  unsigned long long base; float inv_t32, c, kb; uint64_t best; float second;
  __device__ __forceinline__ void init(uint64_t seed, uint32_t step, uint32_t t_id, float T, float key0) {
    base = seed + static_cast<uint64_t>(step) * 0x9E3779B97F4A7C15ull + static_cast<uint64_t>(t_id) * 0xC2B2AE3D27D4EB4Full;
    inv_t32 = __double2float_rn(1.0 / static_cast<double>(T));
    c = 1.44269504f * inv_t32;
    best = 0ull; second = -INFINITY; kb = INFINITY;
    raise(key0);
  }
  __device__ __forceinline__ void raise(float key) {                        // |z c|, |B| 1.44 up to 2^k round to 2^(k-24): far below the slack
    const float b2 = key * 1.44269504f;
    kb = fminf(kb, (23.0f + 0.02f + fabsf(b2) * 4e-6f) - b2);
  }
  __device__ __forceinline__ uint64_t first(int64_t i) const { return base + static_cast<uint64_t>(i) * kHashStep; }   // (i may lie in front of the row)
  __device__ __forceinline__ uint32_t bits(uint32_t i) const { return bits_of(first(i)); }
  static __device__ __forceinline__ uint32_t bits_of(uint64_t x) {
    x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull; x ^= x >> 27; x *= 0x94D049BB133111EBull; x ^= x >> 31;
    return static_cast<uint32_t>(x >> 41) & 0x7FFFFFu;
  }
  // 2^23 exp(z / T - B) + 1: a logit whose 2^23 - h is larger cannot reach B
  __device__ __forceinline__ bool within(float z, uint32_t h) const {
    return 16777216.0f - __uint_as_float(0x4B000000u | h) <= ex2_approx(__fmaf_rn(z, c, kb)) + 1.0f;
  }
  __device__ __forceinline__ void take(float z, uint32_t i, uint32_t h) {
    const float u = (static_cast<float>(h) + 0.5f) * (1.0f / 8388608.0f);
    const float key = __fadd_rn(__fmul_rn(z, inv_t32), -logf(-logf(u)));
    const uint64_t p = pack_best(key, i);
    if (p > best) { if (best) second = fmaxf(second, best_value(best)); best = p; raise(key); } else second = fmaxf(second, key);
  }
  // two logits at once (their hashes are independent chains); z = -inf: none
  __device__ __forceinline__ void offer2(float z0, uint32_t i0, float z1, uint32_t i1) { offer2_bits(z0, i0, bits(i0), z1, i1, bits(i1)); }
  // ... neighbours i, i + 1 whose hashes' arguments (first) are at hand
  __device__ __forceinline__ void offer2_at(float z0, uint64_t x0, float z1, uint64_t x1, uint32_t i) { offer2_bits(z0, i, bits_of(x0), z1, i + 1u, bits_of(x1)); }
  __device__ __forceinline__ void offer2_bits(float z0, uint32_t i0, uint32_t h0, float z1, uint32_t i1, uint32_t h1) {
    bool first = within(z0, h0) && z0 > -INFINITY;
    const bool second_too = within(z1, h1) && z1 > -INFINITY;
#pragma unroll 1
    for (bool more = first || second_too; more;) {                          // (the logarithms' code once)
      take(first ? z0 : z1, first ? i0 : i1, first ? h0 : h1);
      more = first && second_too;
      first = false;
    }
  }
};

// The Gumbel-max draw over a residual r > 0 in the place of exp(z / T): key = ln r + g, the logarithms only where 1 - u <= r exp(-B) leaves room for a key of B (a key
// already seen, less 2e-3 for the rounding of the test).
struct ResidualScan {
  unsigned long long base; float room; uint64_t best;                       // room: 2^23 exp(-B)
  __device__ __forceinline__ void init(uint64_t seed, uint32_t step, uint32_t t_id) {
    base = seed + static_cast<uint64_t>(step) * 0x9E3779B97F4A7C15ull + static_cast<uint64_t>(t_id) * 0xC2B2AE3D27D4EB4Full;
    best = 0ull; room = INFINITY;
  }
  // Four neighbours i .. i + 3 (room is infinite at first; a residual that is not positive has no key).
  __device__ __forceinline__ void offer4(const float (&r)[4], int i) {
    const uint64_t x = base + static_cast<uint64_t>(static_cast<int64_t>(i)) * kHashStep;
    uint32_t h[4], m = 0u;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      h[e] = GumbelScan::bits_of(x + static_cast<uint64_t>(e) * kHashStep);
      if (r[e] > 0.0f && 16777216.0f - __uint_as_float(0x4B000000u | h[e]) <= __fmaf_rn(r[e], room, 1.0f)) m |= 1u << e;
    }
#pragma unroll 1
    for (; m; m &= m - 1u) {                                                // (the logarithms' code once)
      const int e = __ffs(static_cast<int>(m)) - 1;
      const float re = (e & 2) ? ((e & 1) ? r[3] : r[2]) : ((e & 1) ? r[1] : r[0]);
      const uint32_t he = (e & 2) ? ((e & 1) ? h[3] : h[2]) : ((e & 1) ? h[1] : h[0]);
      const float u = (static_cast<float>(he) + 0.5f) * (1.0f / 8388608.0f);
      const uint64_t p = pack_best(__fadd_rn(logf(re), -logf(-logf(u))), static_cast<uint32_t>(i + e));
      if (p > best) best = p;
    }
  }
  // The best key so far of the whole warp bounds what its lanes look at. `before`: what this lane had.
  __device__ __forceinline__ void share(uint64_t before) {
    if (!__any_sync(kFull, best != before)) return;
    room = fminf(room, 8388608.0f * ex2_approx((2e-3f - best_value(warp_max_u64(best))) * 1.44269504f));
  }
};

}  // namespace lm

// What the translation units of the library share on the host side: the error text, the device's size, shared-memory grants.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "../../include/lithos_b200.h"

namespace lm {

inline thread_local char g_cuda_error[256] = "";

inline int cuda_fail(cudaError_t e) {
  std::snprintf(g_cuda_error, sizeof(g_cuda_error), "%s: %s", cudaGetErrorName(e), cudaGetErrorString(e));
  return LM_E_CUDA;
}

inline int sm_count(int* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e);
  static thread_local int cached_dev = -1, cached = 0;
  if (cached_dev != dev) {
    e = cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_fail(e);
    cached_dev = dev;
  }
  *out = cached;
  return LM_OK;
}

// Kernels that need more than 48 KB of shared memory, their static arrays included, must be told so once per device (the attribute belongs to the
// device's copy of the function). They are told whatever they ask for, so that nothing here has to know their arrays; remembered per device and kernel,
// raised when a call needs more.
enum KernelSlot { kSlotFast, kSlotTopk, kSlotTopkOrdered, kSlotGeneric, kSlotVocabLocal, kSlotTileFinish, kSlotSlice, kSlotSliceSmall, kSlotSliceTiny, kSlotSlicedMerge, kSlotHead, kSlotCluster,
                  kSlotArgmax = kSlotCluster + 6,   // (the cluster kernel has six instances, the argmax kernel two)
                  kSlotDraftQ = kSlotArgmax + 2,    // (two instances)
                  kSlotVerify = kSlotDraftQ + 2,    // (twelve)
                  kSlotVerifyGiven = kSlotVerify + 12,   // (four)
                  kSlotCount = kSlotVerifyGiven + 4 };

inline int ensure_dynamic_smem(KernelSlot slot, const void* func, size_t bytes, bool large_clusters = false) {
  constexpr int kMaxDevices = 64;
  static std::mutex mutex;
  static size_t granted[kMaxDevices][kSlotCount] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e);
  std::lock_guard<std::mutex> lock(mutex);
  const bool tracked = dev >= 0 && dev < kMaxDevices;
  if (tracked && bytes <= granted[dev][slot]) return LM_OK;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e != cudaSuccess) return cuda_fail(e);
  if (large_clusters) {                                                     // clusters of up to 16 blocks
    e = cudaFuncSetAttribute(func, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return cuda_fail(e);
  }
  if (tracked) granted[dev][slot] = bytes;
  return LM_OK;
}

// The largest cluster of at most `want` blocks (a power of two) of which `fits` says that the device can hold one; 1 needs no cluster.
template <class Fits> inline int cluster_that_fits(int want, Fits fits) {
  while (want > 1 && !fits(want)) want >>= 1;
  return want;
}

// How many clusters of C such blocks the device (a partition of it, a context limited in its SMs) can hold at once: 16 are beyond what every
// device guarantees, and a cluster lies within one group of SMs. Asked once per device, kernel and C (a power of two up to 16). The kernel has been let
// have `smem`.
inline int clusters_at_once(KernelSlot slot, const void* func, int threads, size_t smem, int C) {
  constexpr int kMaxDevices = 64;
  static std::mutex mutex;
  static int known[kMaxDevices][kSlotCount][5] = {};                        // by log2 C: the number and one more (0: not asked yet)
  int dev = 0, log2 = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return C <= 8 ? 1 : 0;
  for (int c = C; c > 1; c >>= 1) log2++;
  std::lock_guard<std::mutex> lock(mutex);
  if (known[dev][slot][log2]) return known[dev][slot][log2] - 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(C)); cfg.blockDim = dim3(static_cast<unsigned>(threads)); cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(C); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, func, &cfg) != cudaSuccess) { n = 0; (void)cudaGetLastError(); }
  known[dev][slot][log2] = n + 1;
  return n;
}
inline bool cluster_fits(KernelSlot slot, const void* func, int threads, size_t smem, int C) { return clusters_at_once(slot, func, threads, smem, C) > 0; }

// A launch in clusters of C blocks; beside: it may begin while the kernel in front of it in the stream is still at work (programmatic stream
// serialization): its blocks are made ready, set up what needs no device memory, and wait (after_predecessor, common.cuh).
template <class... K, class... A>
inline int launch_stream(bool beside, void (*kernel)(K...), dim3 grid, int threads, size_t smem, int C, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(static_cast<unsigned>(threads)); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[n++].val.programmaticStreamSerializationAllowed = beside ? 1 : 0;
  if (C > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = static_cast<unsigned>(C); attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr; cfg.numAttrs = n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
  return e == cudaSuccess ? LM_OK : cuda_fail(e);
}

// ... of a call of few rows, beside its predecessor: only a grid of no more
// blocks than SMs, or of blocks that need an SM each: placed while others are at work, many small blocks pile up on the SMs that happen to be
// free (512 blocks of 128 threads behind a draft draw: a speculative round 49 us so, 45 behind the predecessor's end). Calls in a row, us per call so / behind the
// predecessor's end: 4 nucleus rows 32.5 / 34.0; probabilities of 4 rows 17.8 / 19.6; one FP32 row with a top_k 12.9 / 16.4 (two launches); a
// speculative round 41.1 / 45.3; 64 FP32 rows with mixed knobs 71.2 / 73.4; the projection of 8 rows 206.9 / 207.7.
template <class... K, class... A>
inline int launch_beside(void (*kernel)(K...), dim3 grid, int threads, size_t smem, int C, cudaStream_t st, A... args) {
  int sms = 0;
  const int rc = sm_count(&sms);
  if (rc != LM_OK) return rc;
  return launch_stream(static_cast<long long>(grid.x) * grid.y <= sms || smem >= 114 * 1024, kernel, grid, threads, smem, C, st, args...);
}

inline size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

struct SampleDev;
struct DraftQDev;
struct VerifyDev;
// cluster.cu: one row per thread-block cluster, every row of the call.
int sample_clusters(const SampleDev& P, int sms, cudaStream_t st, bool few = false);   // few: a call of a few rows with one top_k (LM_STATUS_SLICED_PATH)
int argmax_clusters(const void* logits, int dtype, int rows, int vocab, int64_t row_stride, int32_t* out32, int64_t* out64, cudaStream_t st);
int draft_q_clusters(const DraftQDev& P, int sms, cudaStream_t st);
int verify_rows(const VerifyDev& P, int sms, cudaStream_t st);

}  // namespace lm

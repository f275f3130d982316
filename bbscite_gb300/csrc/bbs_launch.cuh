// bbs_launch.cuh -- templated host launchers shared by the kernel TUs.
#pragma once
#include <algorithm>

#include "bbs_kernels.cuh"

namespace bbs {

// Lets a kernel take `smem` bytes of dynamic shared memory: its limit has to be
// raised where they and its static ones (far below 4 KB in every kernel) are
// more than 48 KB together.  The limit is the kernel's in the whole process, so
// it only ever goes to the most a block may have: set to what a call needs, it
// would take another thread's room between its call here and its launch.
template <typename K>
inline cudaError_t prepare_smem(K kernel, size_t smem) {
  if (smem <= 44 * 1024) return cudaSuccess;
  cudaFuncAttributes at;
  cudaError_t e = cudaFuncGetAttributes(&at, kernel);
  if (e != cudaSuccess || smem <= (size_t)at.maxDynamicSharedSizeBytes) return e;
  int device = 0, block = 0;
  e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = cudaDeviceGetAttribute(&block, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                               device);
  if (e != cudaSuccess) return e;
  if (smem + at.sharedSizeBytes > (size_t)block) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              block - (int)at.sharedSizeBytes);
}

// Persistent launch.  wpc == 1: blocks of `cpb` one-warp chains; wpc > 1:
// blocks of one chain of wpc warps.  As many blocks as chains need, capped
// at what stays resident; each block then walks its chain slots.
template <int W32, int Q, bool SUM, bool REC, int TAB>
int launch_mcmc_k(const RunArgs &a, int cpb, int n_sms, cudaStream_t s) {
  if (a.wpc > 1) cpb = 1;
  const int threads = 32 * a.wpc * cpb;
  if (threads > chain_max_threads(Q)) return (int)cudaErrorInvalidConfiguration;
  const size_t smem = (size_t)a.smem;
  auto kern = mcmc_kernel<W32, Q, SUM, REC, TAB>;
  cudaError_t e = prepare_smem(kern, smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess) return (int)e;
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  const int want = (a.n_chains + cpb - 1) / cpb;
  const int blocks = std::max(1, std::min(want, per_sm * n_sms));
  kern<<<blocks, threads, smem, s>>>(a);
  return (int)cudaGetLastError();
}

template <int W32, int Q, bool SUM, bool REC>
int launch_mcmc_t(const RunArgs &a, int cpb, int n_sms, cudaStream_t s) {
  // (rows of five to eight words replay and trace through the ring)
  // (and the sum score keeps it)
  if constexpr (W32 <= 4 || (!REC && !SUM))
    if (a.chunks > 0) {
      if constexpr (W32 <= 4 && !REC && !SUM)
        if (a.by_counts)
          return launch_mcmc_k<W32, Q, SUM, REC, 2>(a, cpb, n_sms, s);
      return launch_mcmc_k<W32, Q, SUM, REC, 1>(a, cpb, n_sms, s);
    }
  return launch_mcmc_k<W32, Q, SUM, REC, 0>(a, cpb, n_sms, s);
}

// Work-list launch: enough resident slots to fill the GPU, never more than
// there are units.  Blocks of wpb one-warp slots (b.wpc == 1), or of one
// slot of wpb == b.wpc warps.
template <int W32, int Q, bool SUM, bool MULTI, int TAB>
int launch_batch_k(const BatchArgs &b, int wpb, int n_sms, cudaStream_t s) {
  const int threads = 32 * wpb;
  if (threads > chain_max_threads(Q)) return (int)cudaErrorInvalidConfiguration;
  if (b.wpc < 1 || b.wpc > 4 || (b.wpc > 1) != MULTI ||
      (MULTI && wpb != b.wpc))
    return (int)cudaErrorInvalidValue;
  const int slots = wpb / b.wpc;
  const size_t smem = (size_t)b.smem;
  auto kern = batch_kernel<W32, Q, SUM, MULTI, TAB>;
  cudaError_t e = prepare_smem(kern, smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess) return (int)e;
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  const int want = (b.n_units + slots - 1) / slots;
  const int blocks = std::max(1, std::min(want, per_sm * n_sms));
  kern<<<blocks, threads, smem, s>>>(b);
  return (int)cudaGetLastError();
}

template <int W32, int Q, bool SUM, bool MULTI>
int launch_batch_t(const BatchArgs &b, int wpb, int n_sms, cudaStream_t s) {
  if constexpr (W32 <= 4 || !SUM)
    if (b.chunks > 0) {
      if constexpr (W32 <= 4 && !SUM)
        if (b.by_counts)
          return launch_batch_k<W32, Q, SUM, MULTI, 2>(b, wpb, n_sms, s);
      return launch_batch_k<W32, Q, SUM, MULTI, 1>(b, wpb, n_sms, s);
    }
  return launch_batch_k<W32, Q, SUM, MULTI, 0>(b, wpb, n_sms, s);
}

// One unit per row width: launches with recorded moves or a trace (REC) or
// without, and work-list launches of one-warp chains or chains of several
// warps (MULTI).
template <int W, bool REC>
int launch_mcmc_w(const RunArgs &a, int q, bool sum, int cpb, int n_sms,
                  cudaStream_t s);
template <int W, bool MULTI>
int launch_batch_w(const BatchArgs &b, int q, bool sum, int wpb, int n_sms,
                   cudaStream_t s);

}  // namespace bbs

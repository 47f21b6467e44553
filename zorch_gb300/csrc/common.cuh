// Shared host/device helpers: status codes, launch checks, level offsets.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/zc.h"

namespace zc {

#define ZC_TRY(expr)                       \
  do {                                     \
    zc_status _s = (expr);                 \
    if (_s != ZC_OK) return _s;            \
  } while (0)

#define ZC_CUDA(expr)                                  \
  do {                                                 \
    cudaError_t _e = (expr);                           \
    if (_e != cudaSuccess) return zc::cuda_fail(_e);   \
  } while (0)

zc_status cuda_fail(cudaError_t e);
zc_status launch_check();

// Launches a kernel so that it is set up, and stages its constants, while the
// stream's previous kernel ends (programmatic stream serialization): the gap
// between two launches falls from 2.3 us to under 1. Such a kernel calls
// pdl_wait() on every thread before it touches anything that another kernel
// writes or reads, so it is ordered as by a plain launch, and so is whatever
// follows it. It reads no such data through the read-only path (__ldg), which
// assumes no writer during the kernel's whole life.
//
// No kernel lets its successor start before its own CTAs end
// (griddepcontrol.launch_dependents): the successor's CTAs then crowd the few
// SMs that are free first. With it at the start of every kernel a commit of
// 2^13 x 37 at blow-up 8 took 293 us (167 without, 183 with plain launches) and
// the Basefold open of 2^20 x 8 2.02 ms (1.88 and 2.08); in grids of one CTA
// only, 1.90 ms and nothing else faster by more than the runs differ.
template <class... P, class... A>
inline void pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Lets a launch of `kernel` use `smem` bytes of dynamic shared memory. The limit is
// a property of the kernel, shared by all threads: it is always set to the largest
// value (an SM's 227 KB, less `fixed` for the kernel's own arrays), so that no
// thread lowers it between another's call and launch. Up to 48 KB need no limit.
constexpr size_t kSmemMax = 227 * 1024;
template <class... P>
inline zc_status allow_smem(void (*kernel)(P...), size_t smem, size_t fixed = 0) {
  if (smem <= 48 * 1024) return ZC_OK;
  const size_t limit = smem > kSmemMax - fixed ? smem : kSmemMax - fixed;
  ZC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
  return ZC_OK;
}

// Once the previous kernel is complete and its writes are visible.
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A plain load (see pdl_launch).
__device__ __forceinline__ uint32_t gld(const uint32_t* p) { return *p; }

inline bool is_pow2(int64_t x) { return x > 0 && (x & (x - 1)) == 0; }
inline int ilog2(int64_t x) {
  int l = 0;
  while (((int64_t)1 << l) < x) l++;
  return l;
}

// Work items a CTA of the batched (work-list) kernels takes before it retires
// (0: CTAs stay resident until the list is empty). Retiring CTAs let the block
// scheduler start blocks of a higher-priority stream in between, so a small
// served batch does not wait for a large one to drain.
#ifndef ZC_ITEMS_PER_CTA
#define ZC_ITEMS_PER_CTA 8
#endif
constexpr int kItemsPerCta = ZC_ITEMS_PER_CTA;

// Grid of a work-list launch over `total` items: every item is claimed (grid *
// items per CTA >= total), never more CTAs than items; resident CTAs only
// (occ per SM) when CTAs do not retire. A list shorter than kItemsPerCta
// resident waves gets one CTA per item up to a full wave, so that a small
// batch still spreads over every SM.
inline int64_t batch_grid(int64_t total, int occ, int sms) {
  const int64_t wave = (int64_t)(occ > 0 ? occ : 1) * sms;
  int64_t grid = kItemsPerCta > 0 ? (total + kItemsPerCta - 1) / kItemsPerCta : wave;
  if (kItemsPerCta > 0 && grid < wave) grid = total < wave ? total : wave;
  if (grid > total) grid = total;
  return grid < 0x7fffffff ? grid : 0x7fffffff;
}

// log2 of a power of two, on the device.
__device__ __forceinline__ int ilog2_dev(int64_t x) { return 63 - __clzll((long long)x); }

// Digest-layer layout of an arity-2 tree over L leaves: level l (leaf digests
// = level 0, root = level log2 L) starts at node offset 2L - (2L >> l).
__host__ __device__ __forceinline__ int64_t level_offset(int64_t L, int l) {
  return 2 * L - ((2 * L) >> l);
}

__device__ __forceinline__ void store_digest(uint32_t* dst, const uint32_t* d) {
  uint4* p = reinterpret_cast<uint4*>(dst);
  p[0] = make_uint4(d[0], d[1], d[2], d[3]);
  p[1] = make_uint4(d[4], d[5], d[6], d[7]);
}
__device__ __forceinline__ void load_digest(const uint32_t* src, uint32_t* d) {
  const uint4* p = reinterpret_cast<const uint4*>(src);
  uint4 a = p[0], b = p[1];
  d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
  d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}

}  // namespace zc

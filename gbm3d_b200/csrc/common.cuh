// Shared device helpers for the GBM3D sm_100a kernels.
//
// Numerical contract: the library is compiled with --fmad=false, so no a*b+c
// is fused unless a kernel writes fmaf() itself.  Together with IEEE division
// and square root (nvcc defaults) this makes every kernel's float result a
// fixed function of its inputs, reproduced bit for bit by the CPU oracle's
// FP32 mode.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#define GBM3D_MAX_TAPS 16
#define GBM3D_MAX_LEVELS 6

namespace gbm3d {

__host__ __device__ __forceinline__ int pmod(int a, int L) {
  int r = a % L;
  return r < 0 ? r + L : r;
}

// Row (or column) of the image that row r of the reference's search image
// Ipad holds (source/matchBlocksCPU.m:57-61: 2x2 tiling cropped to L+d2,
// then circshift by h=d2/2).  Rows 0..h-1 hold image rows h..2h-1.
__host__ __device__ __forceinline__ int pad_index(int r, int L, int h) {
  return r < h ? r + h : (r - h) % L;
}

// First statement of every kernel that launch_next() launches: wait until the
// kernels before it on the stream are complete and their writes visible, then
// let the next one's CTAs take the slots that this one leaves free.  The pointers
// given are those read through __ldg and the __restrict__ parameters that are read: loads
// that the compiler may take for untouched by the wait and move up.  They leave here with
// a value of unknown origin, so that no such load can be made before the wait.
template <class... P>
__device__ __forceinline__ void begin_after_previous(P&... read_only) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (..., [](auto& p) { asm volatile("" : "+l"(p)::"memory"); }(read_only));
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch with programmatic stream serialisation: the grid may be set up and its
// CTAs made resident while the previous kernel's last ones still run, and each waits at
// begin_after_previous().  Every kernel of a chain waits, so completion is transitive;
// a plain launch, copy or event after it waits for the whole of it as ever.  Of
// the 47 launches of a 128 x 96 call it saves 1.9 us each.
template <class... P, class... Q>
inline void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Q&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  // in a captured graph plain edges: with several lanes the waiting CTAs hold slots
  // that another lane's kernels could use (a batch of ten images: 16.8 against 16.2 ms)
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &capture);
  cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Q>(args)...);  // the caller reads cudaGetLastError()
}

// 4-byte asynchronous global -> shared copy: no register round trip, so all of
// a tile's or a group's loads are in flight together.  The copying thread calls
// cp_async_wait_all() before the barrier (or __syncwarp) that publishes them.
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
// 16 bytes, both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most N of the thread's committed groups are still in flight.
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One axis of a separable filter bank with its nonzero taps in ascending order.
struct Taps {
  int n;
  int k[GBM3D_MAX_TAPS];
  float h[GBM3D_MAX_TAPS];
};

// Analysis (lo, hi) and synthesis (lo, hi) taps of one axis.
struct AxisBank {
  Taps a[2];
  Taps s[2];
};

}  // namespace gbm3d

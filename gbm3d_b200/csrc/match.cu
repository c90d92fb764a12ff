// Block matching — the search of matchBlocksCPU.m:21-116 and matchBlocksWie.m:21-92.
//
// One warp per reference block.  The block's search window (d+d2-1)^2 of the
// padded image sits in shared memory; lane a owns the d2 candidates with row
// offset a (one per column offset b) and streams the window rows a+r past its
// d2 accumulators, so every shared-memory read of a warp touches 32
// consecutive words.  The reference block itself is read from the window
// (it is the candidate at offset (d2/2, d2/2)) by warp-uniform broadcasts.
//
// Distances are exact FP32 sums of squared differences, row-major over the
// block: t = x - y; acc = fmaf(t, t, acc), in scalar instructions, which the
// scheduler spreads over both FP32 pipes (fmaheavy and fmalite); the paired
// f32x2 form of the same operations issues half as many instructions but runs
// on fmaheavy alone and measured 23 % slower.  The K best candidates are the K
// smallest (distance, column-major window index) pairs — the stable order of
// MATLAB's mink — found by a bitwise radix search for the K-th smallest
// distance with warp reductions, then an index-ordered pick among ties.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "kernels.cuh"
#include "match_search.cuh"
#include "tc.cuh"

namespace gbm3d {

namespace {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}
}  // namespace

bool encode_search_map(CUtensorMap* tm, const float* pad, int R, int Q, int P, int box_rows, int box_cols) {
  auto encode = encode_fn();
  if (!encode || (reinterpret_cast<uintptr_t>(pad) & 15) || (P & 3) || R < 1 || Q < 1 || P < R) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)R, (cuuint64_t)Q};
  const cuuint64_t strides[1] = {(cuuint64_t)P * sizeof(float)};
  const cuuint32_t box[2] = {(cuuint32_t)box_rows, (cuuint32_t)box_cols};
  const cuuint32_t es[2] = {1, 1};
  return encode(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(pad), dims, strides, box, es,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Ipad of the reference for a circularly shifted image: rows (m+d2), cols
// (n+d2), column pitch P floats.  spin is the circshift applied to the image.
// A thread writes rows 4 t .. 4 t + 3 of column x as one 16-byte store (P is a
// multiple of 4; rows R .. P-1 of the pitch are never read as image rows).
__global__ void k_make_pad(const float* __restrict__ img, int m, int n, int h, int spin,
                           float* __restrict__ pad, int P, int R, int Q) {
  begin_after_previous(img);
  const int y0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int x = blockIdx.y;
  if (y0 >= P || x >= Q) return;
  // (pad_index(r) - spin) mod L without divisions when h <= L and 0 <= spin <= L
  // (r < L + 2h, so pad_index needs at most one wrap); the general form otherwise
  auto src = [&](int r, int L) {
    if (h <= L && (unsigned)spin <= (unsigned)L) {
      int t = r < h ? r + h : r - h;
      if (t >= L) t -= L;
      t -= spin;
      return t < 0 ? t + L : t;
    }
    return pmod(pad_index(r, L, h) - spin, L);
  };
  const float* col = img + (size_t)src(x, n) * m;
  const float4 v = make_float4(col[src(y0, m)], col[src(y0 + 1, m)], col[src(y0 + 2, m)], col[src(y0 + 3, m)]);
  *reinterpret_cast<float4*>(pad + y0 + (size_t)x * P) = v;
}

// The search of reference g by one warp: win holds win_floats(D + D2 - 1)
// floats of shared memory (128-byte aligned), lst 224 words, mbar the warp's
// mbarrier (phase: its parity).
template <int D, int D2>
__device__ __forceinline__ void match_ref(const MatchArgs& A, const CUtensorMap* tmap, const int g, float* win,
                                          uint32_t* lst, uint64_t* mbar, uint32_t& phase, const int lane) {
  constexpr int WD = D + D2 - 1;  // window rows/cols that candidates touch
  constexpr int WP = win_pitch(WD);
  const int i = g % A.M, j = g / A.M;

  // ---- stage the search window: one TMA copy (this GPU's search image, no
  // multicast) of a WP x WD box whose first row i s is rounded down to a
  // multiple of 4 (a 16-byte aligned coordinate); the window starts o rows
  // into each staged column.  Rows past the search image read as zero.
  const int y0 = i * A.s, o = y0 & 3;
  if (lane == 0) {
    tc::fence_proxy_async();  // this warp's earlier reads of the buffer come first
    tc::mbar_expect_tx(mbar, WP * WD * (int)sizeof(float));
    tc::tma_load_2d(win, tmap, y0 - o, j * A.s, mbar);
  }
  if (!tc::mbar_wait(mbar, phase, MATCH_WAIT_CYCLES)) {
    // the copy did not land in time: give it the full limit again before the
    // buffer is reused, report, and leave this reference's S unwritten
    tc::mbar_wait(mbar, phase, MATCH_WAIT_CYCLES);
    phase ^= 1u;
    if (lane == 0 && A.err) atomicOr(A.err, 4);
    return;
  }
  phase ^= 1u;
  const float* wv = win + o;
  const int count = search_exhaustive<D, D2>(A, wv, lst, lane);
  emit_group<D, D2>(A, g, i, j, wv, lst + 64, count, lane);
}

// Shared memory of a 4-warp CTA: the warps' window buffers, their lst words,
// their mbarriers.
template <int D, int D2>
struct MatchSmem {
  static constexpr int WF = win_floats(D + D2 - 1);
  static constexpr size_t LST = (size_t)4 * WF * sizeof(float);
  static constexpr size_t MBAR = LST + (size_t)4 * 224 * sizeof(uint32_t);
  static constexpr size_t BYTES = MBAR + 4 * sizeof(uint64_t);
};

// WIN: the group window of the strip form (A.g0, A.gn); without it the grid
// covers every group in order.
template <int D, int D2, bool WIN>
__global__ void __launch_bounds__(128, 7) k_match(const __grid_constant__ CUtensorMap tmap, MatchArgs A) {
  begin_after_previous();
  using SM = MatchSmem<D, D2>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = WIN ? window_group(blockIdx.x * 4 + warp, A.g0, A.gn, A.M * A.N) : blockIdx.x * 4 + warp;
  if (WIN ? g < 0 : g >= A.M * A.N) return;  // warp-uniform
  float* win = reinterpret_cast<float*>(smem_raw) + warp * SM::WF;
  uint32_t* lst = reinterpret_cast<uint32_t*>(smem_raw + SM::LST) + warp * 224;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + SM::MBAR) + warp;
  if (lane == 0) {
    tc::mbar_init(mbar, 1);
    tc::fence_mbar_init();
  }
  __syncwarp();
  uint32_t phase = 0;
  match_ref<D, D2>(A, &tmap, g, win, lst, mbar, phase, lane);
}

// Few references of a large patch: a CTA per reference, each warp the distances of
// D2 / 4 candidate columns, warp 0 the selection and the gathers.  One warp per
// reference takes 24 us however few there are at patch 16 (16.4 k instructions of
// exact SSD in a row); split it takes 15 for the 48 of 128 x 96.
template <int D, int D2>
__global__ void __launch_bounds__(128) k_match_split(const __grid_constant__ CUtensorMap tmap, MatchArgs A) {
  begin_after_previous();
  constexpr int WD = D + D2 - 1, WP = win_pitch(WD), NB = D2 / 4;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* win = reinterpret_cast<float*>(smem_raw);
  float* keys = win + win_floats(WD);                                       // [b][lane]
  uint32_t* lst = reinterpret_cast<uint32_t*>(keys + D2 * 32);
  __shared__ uint64_t mbar;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = window_group(blockIdx.x, A.g0, A.gn, A.M * A.N);
  if (g < 0) return;  // the same for the whole CTA
  const int i = g % A.M, j = g / A.M, y0 = i * A.s, o = y0 & 3;
  if (threadIdx.x == 0) {
    tc::mbar_init(&mbar, 1);
    tc::fence_mbar_init();
    tc::mbar_expect_tx(&mbar, WP * WD * (int)sizeof(float));
    tc::tma_load_2d(win, &tmap, y0 - o, j * A.s, &mbar);
  }
  __syncthreads();  // the barrier word is initialised
  const bool ok = tc::mbar_wait(&mbar, 0, MATCH_WAIT_CYCLES);
  if (!__syncthreads_and(ok)) {
    // give the copy the full limit again before the buffer goes away, report
    if (!ok) tc::mbar_wait(&mbar, 0, MATCH_WAIT_CYCLES);
    if (threadIdx.x == 0 && A.err) atomicOr(A.err, 4);
    return;
  }
  const float* wv = win + o;
  float part[NB];
  exact_ssd<D, D2, NB>(wv, lane, warp * NB, part);
#pragma unroll
  for (int b = 0; b < NB; ++b) keys[(warp * NB + b) * 32 + lane] = part[b];
  __syncthreads();
  if (warp) return;
  float acc[D2];
#pragma unroll
  for (int b = 0; b < D2; ++b) acc[b] = keys[b * 32 + lane];
  const int count = select_group<D, D2>(A, wv, acc, lst, lane);
  emit_group<D, D2>(A, g, i, j, wv, lst + 64, count, lane);
}

// List mode: the references A.list[0 .. *A.list_count), grid-stride over the list.
template <int D, int D2>
__global__ void __launch_bounds__(128) k_match_list(const __grid_constant__ CUtensorMap tmap, MatchArgs A) {
  begin_after_previous();
  using SM = MatchSmem<D, D2>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* win = reinterpret_cast<float*>(smem_raw) + warp * SM::WF;
  uint32_t* lst = reinterpret_cast<uint32_t*>(smem_raw + SM::LST) + warp * 224;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + SM::MBAR) + warp;
  if (lane == 0) {
    tc::mbar_init(mbar, 1);
    tc::fence_mbar_init();
  }
  __syncwarp();
  uint32_t phase = 0;
  const int n = *A.list_count;
  for (int t = blockIdx.x * 4 + warp; t < n; t += gridDim.x * 4) {
    const int g = A.list[t];
    if ((unsigned)g < (unsigned)(A.M * A.N)) match_ref<D, D2>(A, &tmap, g, win, lst, mbar, phase, lane);
    __syncwarp();  // the next reference restages win and lst
  }
}

template <int D, int D2, bool WIN>
static cudaError_t launch_match_t(const MatchArgs& A, cudaStream_t st) {
  constexpr int WD = D + D2 - 1;
  const size_t sm = MatchSmem<D, D2>::BYTES;
  CUtensorMap tm;
  if (!encode_search_map(&tm, A.pad, A.R, A.Q, A.P, win_pitch(WD), WD)) return cudaErrorInvalidValue;
  // The attribute belongs to the current device, so it is set before every
  // launch (a host-side call that costs well under a microsecond) rather than
  // remembered once per process: a second device, or another host thread on
  // it, would otherwise launch without it.
  cudaError_t e = cudaFuncSetAttribute(k_match<D, D2, WIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  const int G = A.gn > 0 ? A.gn : A.M * A.N;
  if (A.gn < 0) return cudaSuccess;  // an empty window
  launch_next(k_match<D, D2, WIN>, (G + 3) / 4, 128, sm, st, tm, A);
  return cudaGetLastError();
}

template <int D, int D2>
static cudaError_t launch_match_split(const MatchArgs& A, cudaStream_t st) {
  constexpr int WD = D + D2 - 1;
  const size_t sm = (size_t)(win_floats(WD) + D2 * 32 + 224) * sizeof(float);
  CUtensorMap tm;
  if (!encode_search_map(&tm, A.pad, A.R, A.Q, A.P, win_pitch(WD), WD)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_match_split<D, D2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  if (A.gn < 0) return cudaSuccess;  // an empty window
  launch_next(k_match_split<D, D2>, A.gn > 0 ? A.gn : A.M * A.N, 128, sm, st, tm, A);
  return cudaGetLastError();
}

template <int D, int D2>
static cudaError_t launch_match_list_t(const MatchArgs& A, cudaStream_t st) {
  constexpr int WD = D + D2 - 1;
  const size_t sm = MatchSmem<D, D2>::BYTES;
  CUtensorMap tm;
  if (!encode_search_map(&tm, A.pad, A.R, A.Q, A.P, win_pitch(WD), WD)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_match_list<D, D2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  const int G = A.M * A.N;
  // enough warps for the rare references a list holds; the rest exit at once
  const int blocks = std::min((G + 3) / 4, 2 * 148);
  launch_next(k_match_list<D, D2>, blocks, 128, sm, st, tm, A);
  return cudaGetLastError();
}

cudaError_t launch_match_list(int d, int d2, const MatchArgs& A, cudaStream_t st) {
  if (A.s < 1 || A.s > d || !A.list || !A.list_count) return cudaErrorInvalidValue;
#define GBM3D_MATCHL_CASE(DD, DD2) \
  if (d == DD && d2 == DD2) return launch_match_list_t<DD, DD2>(A, st);
  GBM3D_MATCHL_CASE(8, 16) GBM3D_MATCHL_CASE(8, 24) GBM3D_MATCHL_CASE(8, 32)
#undef GBM3D_MATCHL_CASE
  return cudaErrorInvalidValue;
}

bool match_supported(int d, int d2) {
  return (d == 8 || d == 16 || d == 32) && (d2 == 16 || d2 == 24 || d2 == 32);
}

cudaError_t launch_match(int d, int d2, const MatchArgs& A, cudaStream_t st) {
  if (A.s < 1 || A.s > d) return cudaErrorInvalidValue;
  if (match_bound_supported(d, d2, A)) return launch_match_bound(A, st);
  // patches 16 and 32, at most two references per SM: split.  Both spins of step 1 at patch
  // 16, us unsplit / split: 48 references 75 / 58, 256 77 / 65, 1024 98 / 119, 2304 149 / 168
  // (a split reference keeps three warps waiting for the selection); patch 32: 256 290 / 150,
  // 1024 354 / 415.
  const long groups = A.gn > 0 ? A.gn : (long)A.M * A.N;
#define GBM3D_SPLIT_CASE(DD, DD2) \
  if (d == DD && d2 == DD2 && groups <= 2 * 148) return launch_match_split<DD, DD2>(A, st);
  GBM3D_SPLIT_CASE(16, 16) GBM3D_SPLIT_CASE(16, 24) GBM3D_SPLIT_CASE(16, 32)
  GBM3D_SPLIT_CASE(32, 16) GBM3D_SPLIT_CASE(32, 24) GBM3D_SPLIT_CASE(32, 32)
#undef GBM3D_SPLIT_CASE
#define GBM3D_MATCH_CASE(DD, DD2) \
  if (d == DD && d2 == DD2) return A.gn ? launch_match_t<DD, DD2, true>(A, st) : launch_match_t<DD, DD2, false>(A, st);
  GBM3D_MATCH_CASE(8, 16) GBM3D_MATCH_CASE(8, 24) GBM3D_MATCH_CASE(8, 32)
  GBM3D_MATCH_CASE(16, 16) GBM3D_MATCH_CASE(16, 24) GBM3D_MATCH_CASE(16, 32)
  GBM3D_MATCH_CASE(32, 16) GBM3D_MATCH_CASE(32, 24) GBM3D_MATCH_CASE(32, 32)
#undef GBM3D_MATCH_CASE
  return cudaErrorInvalidValue;
}

// Gather the blocks a match set selects from another image's search image:
// the colour form matches on luma and filters every channel with those sets.
// vol is tile-space (vm = M d rows), block (i, j) slot k at rows i d, cols j d.
// A thread per row and column, rows along the threads, all slots in turn: stores
// are whole lines and d rows share a match index.  The flat version of it
// (divisions of 64-bit indices, stores in d-element pieces) took 162 us for
// 1024^2 x 16; this 33.
template <int D>
__global__ void __launch_bounds__(256) k_gather_volume(const float* __restrict__ pad, int P, int M, int s, int d2,
                                                       int K, const uint32_t* __restrict__ S,
                                                       const int32_t* __restrict__ cnt, float* __restrict__ vol) {
  begin_after_previous(pad, S, cnt);
  // columns along x: a dense grid has more of them than the other grid dimensions hold
  const int y = blockIdx.y * 256 + threadIdx.x, x = blockIdx.x, vm = M * D;
  if (y >= vm) return;
  const int i = y / D, r = y % D, j = x / D, c = x % D, h = d2 / 2;
  const size_t g = i + (size_t)M * j;
  const int nm = cnt ? __ldg(cnt + g) : K;
  const uint32_t* Sg = S + g * K;
  const float* src = pad + (size_t)(i * s + r) + (size_t)(j * s + c) * P;
  float* dst = vol + y + (size_t)vm * x;
  const size_t slot = (size_t)vm * gridDim.x;
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    int e = (int)__ldg(Sg + k) - 1;
    if (k >= nm || (unsigned)e >= (unsigned)(d2 * d2)) e = h + h * d2;
    const int b = d2 == 32 ? e >> 5 : e / d2, a = e - b * d2;
    dst[slot * k] = __ldg(src + a + (size_t)b * P);
  }
}

cudaError_t launch_gather_volume(const float* pad, int P, int M, int N, int s, int d, int d2, int K, const uint32_t* S,
                                 const int32_t* cnt, float* vol, cudaStream_t st) {
  const dim3 grid(N * d, (M * d + 255) / 256);
  switch (d) {
    case 8: launch_next(k_gather_volume<8>, grid, 256, 0, st, pad, P, M, s, d2, K, S, cnt, vol); break;
    case 16: launch_next(k_gather_volume<16>, grid, 256, 0, st, pad, P, M, s, d2, K, S, cnt, vol); break;
    case 32: launch_next(k_gather_volume<32>, grid, 256, 0, st, pad, P, M, s, d2, K, S, cnt, vol); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_make_pad(const float* img, int m, int n, int d2, int spin, float* pad, int P,
                            cudaStream_t st) {
  const int R = m + d2, Q = n + d2;
  dim3 grid((P / 4 + 255) / 256, Q);
  if ((P & 3) || P < R || (reinterpret_cast<uintptr_t>(pad) & 15)) return cudaErrorInvalidValue;
  launch_next(k_make_pad, grid, 256, 0, st, img, m, n, d2 / 2, spin, pad, P, R, Q);
  return cudaGetLastError();
}

}  // namespace gbm3d

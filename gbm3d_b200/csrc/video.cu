// Video: block matching across a window of frames and aggregation into the
// frames — matchBlocksV.m:21-116 (top-K branch) and the aggregation loop of
// denoiseAndAggregateV.m:59-89.  The 3D wavelet hard threshold between them
// is the step-1 one (wavelet.cu) with the video's filter bank.
#include "common.cuh"
#include "kernels.cuh"

namespace gbm3d {

namespace {

// One CTA per reference block of the centre frame (stride d).  For every
// frame f of the window, the 2d x 2d window of that frame's search image is
// staged in shared memory and the exact FP32 SSD of each of the d x d
// candidate offsets is computed in row-major order (t = ref - cand,
// acc = fmaf(t, t, acc)).  Keys (distance bits << 32 | index a + b d + f d^2)
// sit in shared memory; the K smallest are taken in K rounds of a block-wide
// minimum (the stable (value, index) order of mink).  S(1) is the reference.
template <int D>
__global__ void __launch_bounds__(128) k_match_video(VideoMatchArgs A) {
  begin_after_previous();
  constexpr int WD = 2 * D, H = D / 2, DD = D * D;
  extern __shared__ unsigned long long keys[];   // F * D^2
  float* win = reinterpret_cast<float*>(keys + A.F * DD);  // WD x WD, column-major
  float* xr = win + WD * WD;                               // reference block, row-major
  __shared__ unsigned long long red[4];
  __shared__ uint32_t sel[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = blockIdx.x, i = g % A.M, j = g / A.M;
  if (A.redo && !A.redo[g]) return;  // the bounded matcher has done it
  const int ref = (A.F - 1) / 2;
  const int nc = A.F * DD;
  {  // the reference block: offset (d/2, d/2) of the centre frame's window
    const float* pr = A.pads[ref];
    for (int e = tid; e < DD; e += 128) {
      const int r = e / D, c = e % D;
      xr[e] = pr[(size_t)(i * D + H + r) + (size_t)(j * D + H + c) * A.P];
    }
  }
  for (int f = 0; f < A.F; ++f) {
    const float* pad = A.pads[f];
    __syncthreads();
    for (int e = tid; e < WD * WD; e += 128) {
      const int r = e % WD, c = e / WD;
      win[e] = pad[(size_t)(i * D + r) + (size_t)(j * D + c) * A.P];
    }
    __syncthreads();
    if constexpr (D == 32) {
      // 1024 candidates, 8 per thread: lane a = candidate row, warp w the
      // columns b = 8w .. 8w+7.  Per pixel (r, c) the reference value is one
      // broadcast and the 8 candidates' window values slide along the row
      // a + r in registers (one new shared load per c), so the loop runs at
      // the FP32 issue rate instead of two shared loads per FMA.  Each
      // candidate still accumulates in the order (r, then c).
      constexpr int NB = 8;
      const int a = tid & 31, b0 = (tid >> 5) * NB;
      float acc[NB];
#pragma unroll
      for (int q = 0; q < NB; ++q) acc[q] = 0.f;
      for (int r = 0; r < D; ++r) {
        const float* wr = win + (a + r) + b0 * WD;  // row a + r of the window, from column b0
        const float4* x4p = reinterpret_cast<const float4*>(xr + r * D);
        float wv[NB];  // wv[j & 7] = window column b0 + j of this row
#pragma unroll
        for (int q = 0; q < NB - 1; ++q) wv[q] = wr[q * WD];
#pragma unroll
        for (int c4 = 0; c4 < D / 4; ++c4) {
          const float4 x4 = x4p[c4];
          const float xs[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int c = c4 * 4 + u;
            wv[(c + NB - 1) & (NB - 1)] = wr[(c + NB - 1) * WD];
#pragma unroll
            for (int q = 0; q < NB; ++q) {
              const float t = xs[u] - wv[(c + q) & (NB - 1)];
              acc[q] = fmaf(t, t, acc[q]);
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        const uint32_t idx = (uint32_t)(a + (b0 + q) * D + f * DD);
        keys[idx] = ((unsigned long long)__float_as_uint(acc[q]) << 32) | idx;
      }
    } else {
      for (int cand = tid; cand < DD; cand += 128) {
        const int a = cand % D, b = cand / D;
        float acc = 0.f;
        for (int r = 0; r < D; ++r)
#pragma unroll 8
          for (int c = 0; c < D; ++c) {
            const float t = xr[r * D + c] - win[(a + r) + (b + c) * WD];
            acc = fmaf(t, t, acc);
          }
        const uint32_t idx = (uint32_t)(a + b * D + f * DD);
        keys[idx] = ((unsigned long long)__float_as_uint(acc) << 32) | idx;
      }
    }
  }
  __syncthreads();
  // K rounds of a block-wide minimum over the keys
  for (int k = 0; k < A.K; ++k) {
    unsigned long long best = ~0ull;
    for (int e = tid; e < nc; e += 128) best = min(best, keys[e]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (tid == 0) {
      const unsigned long long b = min(min(red[0], red[1]), min(red[2], red[3]));
      sel[k] = (uint32_t)(b & 0xffffffffu);
      keys[sel[k]] = ~0ull;
    }
    __syncthreads();
  }
  if (tid == 0) sel[0] = (uint32_t)(DD * A.F / 2 + H);  // S(1) = d^2 F/2 + d/2 + 1 (matchBlocksV.m:103), 0-based
  __syncthreads();
  for (int k = tid; k < A.K; k += 128) A.S[(size_t)g * A.K + k] = sel[k] + 1;
  // Volume(i d + r, j d + c, k): the selected block, image-shaped m x n x K
  const size_t mn = (size_t)A.m * A.n;
  for (int e = tid; e < A.K * DD; e += 128) {
    const int k = e / DD, r = e % D, c = (e / D) % D;
    const uint32_t s = sel[k];
    const int a = (int)(s % D), b = (int)((s / D) % D), f = (int)(s / DD);
    A.volume[(size_t)(i * D + r) + (size_t)A.m * (j * D + c) + mn * k] =
        A.pads[f][(size_t)(i * D + a + r) + (size_t)(j * D + b + c) * A.P];
  }
}

// Owner-computes aggregation into the F frames.  A CTA owns VT x VT pixels of one
// frame: it lists the blocks (reference y, x, slot k) of that frame that touch
// them, in the reference's loop order (block k of (y, x) starts at (a + y d - d/2,
// b + x d - d/2) of frame f and is skipped when the start is negative), and every
// thread steps through the list for its four pixels of one row; each term fl(w block)
// is added in double (the reference's U and out.K are double arrays).  A thread
// per pixel testing every (reference, slot) pair of its neighbourhood took 233 us
// for three 720p frames; this 67 (entries' loads four at a time ahead of the adds: 77).  A list that could overflow is applied and
// refilled, so any capacity gives the same sums.
//   With Y, the sums are added to the call's single-precision accumulators, as
// VBM3D.m:52-56 does after each window, instead of being written out.
constexpr int VT = 32, VTHREADS = 256, VLIST = 512;

template <int D>
__global__ void __launch_bounds__(VTHREADS) k_aggregate_video(VideoAggArgs A) {
  const uint32_t* Sg = A.S;
  const float* wgt = A.wgt;
  const float* vsum = A.vsum;
  begin_after_previous(Sg, wgt, vsum);
  constexpr int H = D / 2;
  __shared__ int4 lst[VLIST];
  __shared__ int wcnt[VTHREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R0 = blockIdx.x * VT, C0 = blockIdx.y * VT, fr = blockIdx.z, K = A.K;
  const size_t mn = (size_t)A.m * A.n;
  // references whose blocks can touch the tile: y D - H <= R0 + VT - 1 and y D + H - 1 + D > R0
  const int ylo = max(0, (R0 - H - D + 1 + 4 * D) / D - 4), yhi = min(A.M - 1, (R0 + VT - 1 + H) / D);
  const int xlo = max(0, (C0 - H - D + 1 + 4 * D) / D - 4), xhi = min(A.N - 1, (C0 + VT - 1 + H) / D);
  const int ny = yhi - ylo + 1, nx = xhi - xlo + 1, total = ny > 0 && nx > 0 ? ny * nx * K : 0;
  // pixels: row lane, columns warp + 8 q
  double u[4] = {0.0, 0.0, 0.0, 0.0}, w[4] = {0.0, 0.0, 0.0, 0.0};
  auto apply = [&](int count) {
    for (int e = 0; e < count; ++e) {
      const int4 en = lst[e];
      const int rr = lane - (short)(en.x & 0xffff), cc0 = warp - (en.x >> 16);
      const float wg = __int_as_float(en.z);
      const double dw = (double)wg;
      const float* src = vsum + (((size_t)(unsigned)en.w << 32) | (unsigned)en.y) + rr;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int cc = cc0 + 8 * q;
        if ((unsigned)cc < (unsigned)D && (unsigned)rr < (unsigned)D) {
          u[q] += (double)(wg * __ldg(src + (unsigned)(A.m * cc)));
          w[q] += dw;
        }
      }
    }
  };
  int n = 0;
  for (int base = 0; base < total; base += VTHREADS) {
    const int t = base + tid;
    bool hit = false;
    int4 en = make_int4(0, 0, 0, 0);
    if (t < total) {
      const int k = t % K, yx = t / K, y = ylo + yx / nx, x = xlo + yx % nx, g = y + A.M * x;
      const int e = (int)__ldg(Sg + (size_t)g * K + k) - 1;
      const int a = e % D, b = (e / D) % D, f = e / (D * D);
      const int r = a + y * D - H, c = b + x * D - H;
      hit = f == fr && r >= 0 && c >= 0 && r < R0 + VT && r + D > R0 && c < C0 + VT && c + D > C0;
      if (hit) {
        en.x = ((r - R0) & 0xffff) | ((c - C0) << 16);
        const size_t o = (size_t)(y * D) + (size_t)A.m * (x * D) + mn * k;
        en.y = (int)(unsigned)o;
        en.w = (int)(o >> 32);
        en.z = __float_as_int(__ldg(wgt + g));
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wcnt[warp] = __popc(bal);
    __syncthreads();
    int off = n, tot = 0;
#pragma unroll
    for (int v = 0; v < VTHREADS / 32; ++v) {
      off += v < warp ? wcnt[v] : 0;
      tot += wcnt[v];
    }
    if (hit) lst[off + __popc(bal & ((1u << lane) - 1u))] = en;
    n += tot;
    __syncthreads();
    if (n > VLIST - VTHREADS) {
      apply(n);
      n = 0;
      __syncthreads();
    }
  }
  apply(n);
  const int r = R0 + lane;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int c = C0 + warp + 8 * q;
    if (r < A.m && c < A.n) {
      const size_t o = mn * fr + r + (size_t)A.m * c;
      if (A.Y) {
        A.Y[o] = (float)((double)A.Y[o] + u[q]);  // the reference's Y and nn are single arrays
        A.nn[o] = (float)((double)A.nn[o] + w[q]);
      } else {
        A.U[o] = u[q];
        A.W[o] = w[q];
      }
    }
  }
}

}  // namespace

bool video_match_supported(int d, int F, int K) {
  return (d == 8 || d == 16 || d == 32) && F >= 1 && (F & 1) && F <= 31 && K >= 1 && K <= 32 && F * d * d >= K &&
         (size_t)F * d * d * 8 + (size_t)(4 * d * d + d * d) * 4 <= 200 * 1024;
}

cudaError_t launch_match_video(int d, const VideoMatchArgs& B, cudaStream_t st) {
  VideoMatchArgs A = B;
  if (!video_match_supported(d, A.F, A.K)) return cudaErrorInvalidValue;
  if (video_bound_supported(d, A)) {
    const cudaError_t e = launch_match_video_bound(A, st);
    if (e != cudaSuccess) return e;
  } else {
    A.redo = nullptr;
  }
  const size_t sm = (size_t)A.F * d * d * 8 + (size_t)(4 * d * d + d * d) * 4;
  const int G = A.M * A.N;
#define GBM3D_VM_CASE(DD)                                                                                   \
  if (d == DD) {                                                                                            \
    cudaError_t e = cudaFuncSetAttribute(k_match_video<DD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm); \
    if (e != cudaSuccess) return e;                                                                         \
    launch_next(k_match_video<DD>, G, 128, sm, st, A);                                                      \
    return cudaGetLastError();                                                                              \
  }
  GBM3D_VM_CASE(8) GBM3D_VM_CASE(16) GBM3D_VM_CASE(32)
#undef GBM3D_VM_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_aggregate_video(const VideoAggArgs& A, cudaStream_t st) {
  const dim3 grid((A.m + VT - 1) / VT, (A.n + VT - 1) / VT, A.F);
  switch (A.d) {
    case 8: launch_next(k_aggregate_video<8>, grid, VTHREADS, 0, st, A); break;
    case 16: launch_next(k_aggregate_video<16>, grid, VTHREADS, 0, st, A); break;
    case 32: launch_next(k_aggregate_video<32>, grid, VTHREADS, 0, st, A); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace gbm3d

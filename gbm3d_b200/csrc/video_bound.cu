// Video block matching at patch 32 (matchBlocksV.m:21-116, top-K branch) with f16
// tensor-core distances as a bound.
//
// The direct kernel (k_match_video<32>, video.cu) computes all 1024 F distances of a
// reference exactly, 196 k warp instructions at F = 3, of which 16 are kept.  As in
// match_bound.cu the cross terms of all 32 x 32 offsets of a frame are products of the
// window's columns with Toeplitz matrices of the reference's columns (here 40
// rows deep: two m16n8k16 and one m16n8k8 per column and tile), norms come from
// suffix and prefix sums, candidate_threshold() (bound.cuh) keeps every candidate
// that the exact ranking could take, and those are ranked by the exact SSD in
// the direct kernel's operation order.
//   One CTA of four warps per reference; frames pass one after another through
// one window buffer (33 KB: six CTAs per SM), the distances stay in registers,
// and the frames that hold candidates are staged once more for the exact SSD.
//   720p, F = 3: 307 -> 130 us per window; 17.5 k shared-memory wavefronts per
// reference (4.6 k ldmatrix, 7 k the exact SSDs), barriers while one warp ranks.  The
// 32 row and column sums of a thread cross barriers in registers, and some spill (F = 3: 56
// bytes of stores at the 80 registers that six CTAs allow).
// References whose list overflows, or whose values leave the f16 range, are
// marked in A.redo for the direct kernel.
#include "bound.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "tc.cuh"

namespace gbm3d {

namespace {

constexpr int D = 32, DD = D * D, H = D / 2, WD = 2 * D;  // patch, candidates per frame, half, window side
constexpr int WP = 68;                                    // fp32 window pitch
constexpr int HP = 72;                                    // f16 window pitch: ldmatrix rows on distinct banks
constexpr int XP = 48;                                    // a reference column: 8 zeros, 32 values, 8 zeros
constexpr int SP = 65, NP = 36;                           // pitches of the row sums and of the norms
constexpr int LCAND = 256;                                // candidates a list holds
constexpr size_t OFF_W16 = (size_t)WD * WP * sizeof(float);
constexpr size_t OFF_XZ = OFF_W16 + (size_t)WD * HP * sizeof(__half);
constexpr size_t VB_BYTES = OFF_XZ + (size_t)D * 2 * XP * sizeof(__half);
static_assert(2 * D * SP <= WD * WP && D * NP <= WD * WP, "row sums and norms reuse the window");
static_assert(DD * 4 + LCAND * 8 <= WD * HP * 2, "reference block and list reuse the f16 window");

__device__ __forceinline__ float block_sum(float v, float* red, int warp, int lane) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return (red[0] + red[1]) + (red[2] + red[3]);
}

template <int F, int OCC>
__global__ void __launch_bounds__(128, OCC) k_match_video_bound(VideoMatchArgs A) {
  begin_after_previous();
  extern __shared__ __align__(16) unsigned char vsm[];
  float* win = reinterpret_cast<float*>(vsm);               // [column][row]
  __half* w16 = reinterpret_cast<__half*>(vsm + OFF_W16);   // centred f16 window, [column][row]
  __half* xz = reinterpret_cast<__half*>(vsm + OFF_XZ);     // reference columns, twice: [c][shifted by 0, 1][XP]
  float* hs = win;                                          // row sums of columns b .. 31 and 32 .. b + 31
  float* hp = win + D * SP;
  float* nrm = win;                                         // ||w16||^2, [b][a]
  __shared__ float red[4], mx[128], Tsh;
  __shared__ int cnt, cntf[F];
  __shared__ uint32_t sel[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = blockIdx.x, i = g % A.M, j = g / A.M, K = A.K;

  // one 64 x 64 window by 16-byte copies
  auto stage = [&](int f) {
    const float* src = A.pads[f] + (size_t)(i * D) + (size_t)(j * D) * A.P;
#pragma unroll
    for (int q = 0; q < WD * WD / 4 / 128; ++q) {
      const int e = tid + 128 * q, c = e >> 4, r = 4 * (e & 15);
      cp_async16(win + c * WP + r, src + r + (size_t)c * A.P);
    }
    cp_async_wait_all();
    __syncthreads();
  };

  // ---- the reference block: mean, f16 columns, norm
  float m0, nx;
  {
    const float* src = A.pads[(F - 1) / 2] + (size_t)(i * D + H) + (size_t)(j * D + H) * A.P;
    float x[DD / 128], s = 0.f;
#pragma unroll
    for (int q = 0; q < DD / 128; ++q) {
      x[q] = src[lane + (size_t)(warp + 4 * q) * A.P];
      s += x[q];
    }
    m0 = block_sum(s, red, warp, lane) * (1.f / DD);
    s = 0.f;
    for (int e = tid; e < D * 2 * XP; e += 128) xz[e] = __float2half(0.f);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < DD / 128; ++q) {
      const __half h = __float2half_rn(x[q] - m0);
      __half* d = xz + (size_t)(warp + 4 * q) * 2 * XP;
      d[8 + lane] = h;
      d[XP + 7 + lane] = h;
      const float v = __half2float(h);
      s += v * v;
    }
    nx = block_sum(s, red, warp, lane);
  }
  if (tid == 0) cnt = 0;
  if (tid < F) cntf[tid] = 0;

  // ---- distances: warp (mt, p) makes candidate columns b = 16 mt .. + 15 and rows a = 16 p .. + 15
  const int mt = warp & 1, p = warp >> 1, gq = lane >> 2, t = lane & 3;
  const uint32_t adr = tc::smem_u32(w16) +
                       (uint32_t)(((16 * mt + (lane & 7) + 8 * ((lane >> 3) & 1)) * HP + 16 * p + 8 * (lane >> 4)) * 2);
  // B(k, n) = x(k - n): the pair k = 8 kb + 2t, + 1 of column n = lane / 4; the copy shifted
  // by one serves the odd n
  const uint32_t* xb = reinterpret_cast<const uint32_t*>(xz + (gq & 1) * XP) + ((8 + 2 * t - gq - (gq & 1)) >> 1);
  float acc[F][2][4];
  bool big = false;
#pragma unroll
  for (int f = 0; f < F; ++f) {
    __syncthreads();  // the previous frame's norms and f16 window are used up
    stage(f);
    // rounded window; row sums of squares: suffixes of columns 31 .. 0, prefixes of columns 32 .. 62
    const int row = tid & 63, part = tid >> 6;
    float q[D];
    {
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < D; ++u) {
        const int c = part ? D + u : D - 1 - u;
        const __half h = __float2half_rn(win[c * WP + row] - m0);
        w16[c * HP + row] = h;
        const float v = __half2float(h);
        big |= !(fabsf(v) < 60000.f);
        if (part) q[u] = s;  // columns 32 .. 31 + u
        s += v * v;
        if (!part) q[D - 1 - u] = s;
      }
    }
    __syncthreads();
    {
      float* d = (part ? hp : hs) + row;
#pragma unroll
      for (int b = 0; b < D; ++b) d[b * SP] = q[b];
    }
    __syncthreads();
    // column sums the same way: warp 0 rows 31 .. 0, warp 1 rows 32 .. 62 (lane = b)
    if (warp < 2) {
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < D; ++u) {
        const int r = lane * SP + (warp ? D + u : D - 1 - u);
        const float h = hs[r] + hp[r];
        if (warp) q[u] = s;
        s += h;
        if (!warp) q[D - 1 - u] = s;
      }
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int a = 0; a < D; ++a) nrm[lane * NP + a] = q[a];
    }
    __syncthreads();
    if (warp == 1) {
#pragma unroll
      for (int a = 0; a < D; ++a) nrm[lane * NP + a] += q[a];
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[f][nt][e] = 0.f;
#pragma unroll 4
    for (int c = 0; c < D; ++c) {
      uint32_t a[3][4], b[5];  // window rows 16 p .. + 47 in eights, {b 0..7, b 8..15}
#pragma unroll
      for (int u = 0; u < 3; ++u) ldsm4(a[u], adr + c * HP * 2 + 32 * u);
#pragma unroll
      for (int kb = 0; kb < 5; ++kb) b[kb] = xb[c * XP + 4 * kb];
      mma_f16(acc[f][0], a[0][0], a[0][1], a[0][2], a[0][3], b[0], b[1]);
      mma_f16(acc[f][1], a[0][2], a[0][3], a[1][0], a[1][1], b[0], b[1]);
      mma_f16(acc[f][0], a[1][0], a[1][1], a[1][2], a[1][3], b[2], b[3]);
      mma_f16(acc[f][1], a[1][2], a[1][3], a[2][0], a[2][1], b[2], b[3]);
      mma_f16_k8(acc[f][0], a[2][0], a[2][1], b[4]);
      mma_f16_k8(acc[f][1], a[2][2], a[2][3], b[4]);
    }
    __syncthreads();  // the norms are complete
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        acc[f][nt][e] -= 0.5f * nrm[(16 * mt + gq + 8 * (e >> 1)) * NP + 16 * p + 8 * nt + 2 * t + (e & 1)];
  }

  // ---- threshold: the K-th best of the 128 threads' maxima
  float m1 = acc[0][0][0];
#pragma unroll
  for (int f = 0; f < F; ++f)
#pragma unroll
    for (int e = 0; e < 8; ++e) m1 = fmaxf(m1, acc[f][e >> 2][e & 3]);
  mx[tid] = m1;
  big = __syncthreads_or(big);
  {
    int rank = 0;
#pragma unroll 8
    for (int u = 0; u < 128; ++u) rank += mx[u] > m1 || (mx[u] == m1 && u < tid) ? 1 : 0;
    if (rank == K - 1) Tsh = m1;
  }
  float* xrow = reinterpret_cast<float*>(w16);          // reference block, row-major
  uint2* list = reinterpret_cast<uint2*>(xrow + DD);    // (key, index)
  {
    const float* src = A.pads[(F - 1) / 2] + (size_t)(i * D + H) + (size_t)(j * D + H) * A.P;
    for (int e = tid; e < DD; e += 128) xrow[(e & 31) * D + (e >> 5)] = src[(e & 31) + (size_t)(e >> 5) * A.P];
  }
  __syncthreads();
  if (!big) {
    const float th = 0.5f * (nx - candidate_threshold<Bound32>(nx - 2.f * Tsh, nx));
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (acc[f][e >> 2][e & 3] >= th) {
          const int a = 16 * p + 8 * (e >> 2) + 2 * t + (e & 1), b = 16 * mt + gq + 8 * ((e >> 1) & 1);
          const int pos = atomicAdd(&cnt, 1);
          atomicAdd(&cntf[f], 1);
          if (pos < LCAND) list[pos].y = (uint32_t)(a + b * D + f * DD);
        }
  }
  __syncthreads();
  const int C = cnt;
  const bool redo = big || C < K || C > LCAND;
  const size_t mn = (size_t)A.m * A.n;
  if (redo) {
    // an overflow may be windows of one value (black bars, a mask): every distance is exactly
    // zero and the lowest indices win
    const float w0 = A.pads[0][(size_t)(i * D) + (size_t)(j * D) * A.P];
    bool same = !big;  // the same for every thread
    for (int f = 0; f < F && same; ++f) {
      stage(f);
      bool differs = false;
      for (int e = tid; e < WD * WD; e += 128)
        differs |= __float_as_uint(win[(e >> 6) * WP + (e & 63)]) != __float_as_uint(w0);
      same = !__syncthreads_or(differs);
    }
    if (tid == 0) A.redo[g] = same ? 0 : 1;
    if (same) {
      if (tid < K) A.S[(size_t)g * K + tid] = (uint32_t)(tid == 0 ? DD * F / 2 + H : tid) + 1;
      for (int e = tid; e < K * DD; e += 128)
        A.volume[(size_t)(i * D + e % D) + (size_t)A.m * (j * D + (e / D) % D) + mn * (e / DD)] = w0;
    }
    return;
  }
  if (tid == 0) A.redo[g] = 0;

  // ---- exact SSD of the candidates, frame by frame, in the direct kernel's
  // operation order (row-major, t = x - w, acc = fmaf(t, t, acc))
  for (int f = 0; f < F; ++f) {
    if (cntf[f] == 0) continue;  // the same for every thread
    stage(f);
    for (int q = tid; q < C; q += 128) {
      const int ix = (int)list[q].y;
      if (ix >> 10 != f) continue;
      const float* wc = win + (ix & 31) + ((ix >> 5) & 31) * WP;
      float d = 0.f;
      for (int r = 0; r < D; ++r) {
#pragma unroll
        for (int c4 = 0; c4 < D / 4; ++c4) {
          const float4 x4 = reinterpret_cast<const float4*>(xrow + r * D)[c4];
          const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float e = x[u] - wc[r + (4 * c4 + u) * WP];
            d = fmaf(e, e, d);
          }
        }
      }
      list[q].x = __float_as_uint(d);
    }
    __syncthreads();
  }
  // ---- rank by (distance, index); S(1) = d^2 F/2 + d/2 + 1 (matchBlocksV.m:103)
  for (int q = tid; q < C; q += 128) {
    const uint2 me = list[q];
    const unsigned long long mk = ((unsigned long long)me.x << 32) | me.y;
    int rank = 0;
#pragma unroll 4
    for (int u = 0; u < C; ++u) {
      const uint2 ot = list[u];
      rank += (((unsigned long long)ot.x << 32) | ot.y) < mk ? 1 : 0;
    }
    if (rank < K) sel[rank] = rank == 0 ? (uint32_t)(DD * F / 2 + H) : me.y;
  }
  __syncthreads();
  if (tid < K) A.S[(size_t)g * K + tid] = sel[tid] + 1;
  // Volume(i d + r, j d + c, k): the selected block, image-shaped m x n x K
  for (int e = tid; e < K * DD; e += 128) {
    const int k = e / DD, r = e % D, c = (e / D) % D;
    const uint32_t s = sel[k];
    const int a = (int)(s % D), b = (int)((s / D) % D), f = (int)(s / DD);
    A.volume[(size_t)(i * D + r) + (size_t)A.m * (j * D + c) + mn * k] =
        __ldg(A.pads[f] + (size_t)(i * D + a + r) + (size_t)(j * D + b + c) * A.P);  // address from shared memory
  }
}

template <int F, int OCC>
cudaError_t launch_vb(const VideoMatchArgs& A, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_match_video_bound<F, OCC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VB_BYTES);
  if (e != cudaSuccess) return e;
  launch_next(k_match_video_bound<F, OCC>, A.M * A.N, 128, VB_BYTES, st, A);
  return cudaGetLastError();
}

}  // namespace

// Windows of 3 to 11 frames (8 F distances per thread stay in registers).
bool video_bound_supported(int d, const VideoMatchArgs& A) {
  return d == D && A.redo && A.F >= 3 && A.F <= 11 && A.K <= 32 && (A.P & 3) == 0;
}

cudaError_t launch_match_video_bound(const VideoMatchArgs& A, cudaStream_t st) {
  switch (A.F) {
    case 3: return launch_vb<3, 6>(A, st);
    case 5: return launch_vb<5, 5>(A, st);
    case 7: return launch_vb<7, 4>(A, st);
    case 9: return launch_vb<9, 3>(A, st);
    case 11: return launch_vb<11, 3>(A, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gbm3d

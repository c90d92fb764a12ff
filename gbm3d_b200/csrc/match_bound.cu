// Block matching at patch 8 and a 32 x 32 search: tensor-core distances bound
// the candidates, the exact FP32 SSD ranks them (matchBlocksCPU.m:21-116,
// matchBlocksWie.m:21-92, top-K branch).
//
// The exhaustive matcher (match.cu) spends 4096 of its 5.7 k warp instructions
// per reference on the exact SSD of 1024 candidates, of which 16 are kept.
// Here a reference's distances come from 64 mma.sync m16n8k16 (f16 operands,
// FP32 sums): the cross terms <x, w> of all 32 x 32 offsets are, per block
// column c, a product of the window's columns (A: row b = candidate column,
// k = window row) with a Toeplitz matrix of the reference's column
// (B(k, n) = x(k - n, c)), so the window is read as it lies, with no im2col
// copy, and a lane builds its B fragment from two values.  The legacy warp
// MMA is the right unit here: a reference needs 32 x 32 x 8 x 8 useful
// products, four warps share one staged window, and the accumulators are
// consumed by the warp that made them; the tcgen05 version (match_tc.cu) needs
// tile-wide barriers and TMEM round trips around its selection and is slower.
//
// The bound itself, candidate_threshold(), is derived in bound.cuh.  The candidates
// it leaves are listed and ranked by the exact SSD and index, as the exhaustive
// matcher ranks.
//
// A CTA takes four references of one grid row (i; j .. j + 3): their windows
// overlap, so the union (39 x (3 s + 39)) is staged by one TMA copy, rounded to
// f16 once and its 8 x 8 norm sums made once.  Tiles along j keep the row
// offset common, so each warp's MMA operands start on a 16-byte boundary
// (ldmatrix) at every stride.
//
// Measured against the exhaustive matcher (B200, both steps of one call):
// 4096^2 at strides 8 / 7 3.29 -> 1.80 ms, dense (stride 3, two spins) 40.1 ->
// 21.3 ms, 1677 x 1531 at stride 3 4.73 -> 2.4 ms.  About 1.8 k warp instructions
// per reference instead of 5.7 k; bound by the shared-memory pipe (82-92 % of the
// cycles: 570-720 wavefronts per reference, of them 160 ldmatrix, about 165 exact-SSD
// loads of scattered candidates, 85 + 40 for the rounded window and the norm sums), not by
// issue (56-60 %).
//   Where the list overflows the bound is paid on top of the exhaustive search, so
// windows of one value, whose distances are all zero, are told from the rest there
// (2048^2 at strides 8 / 6, both steps: a flat image 1.79 -> 1.26 ms, the exhaustive matcher
// 1.29; one half masked 1.32 -> 0.63 against 1.33; noisy 0.55 against 1.05).
#include <cuda.h>
#include <cuda_fp16.h>

#include "bound.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "match_search.cuh"
#include "tc.cuh"

namespace gbm3d {

namespace {

constexpr int D = 8, D2 = 32, H = D2 / 2, WD = D + D2 - 1;  // patch, search side, its half, window side
constexpr int NREF = 4;                                     // references (warps) per CTA
constexpr int WP = win_pitch(WD);                           // pitch of the staged window and of the norm sums
constexpr int MAXCH = (3 * D + D2 + 7) / 8;                 // chunks of 8 window positions along j at stride 8
constexpr int MAXCOL = 8 * MAXCH + 7;                       // staged columns at stride 8
constexpr int HP = 40;                                      // f16 pitch: 80 bytes, ldmatrix rows on distinct banks
constexpr int LCAND = 128;                                  // candidates a warp's list holds
// 32-bit words of a warp's scratch: the exhaustive search's 224, or 64 (reference
// block, row-major) + 32 (S) + 2 LCAND (keys and indices)
constexpr int SCR = 96 + 2 * LCAND;

// Whether a reference's window holds one value throughout.  A call, and only where the whole window is
// within the bound: inlined it costs every reference 1 % by the code around it.
__device__ __noinline__ bool one_value(const float* wv, int lane) {
  uint32_t differs = 0;
#pragma unroll 1
  for (int c = 0; c < WD; ++c)
    differs |= (__float_as_uint(wv[c * WP + lane]) ^ __float_as_uint(wv[0])) |
               (__float_as_uint(wv[c * WP + WD - 32 + lane]) ^ __float_as_uint(wv[0]));
  return !__any_sync(0xffffffffu, differs);
}

// Groups of the column range [j0, j0 + nj): blockIdx.x = i + M (tile of four columns).
__global__ void __launch_bounds__(128, 6) k_match_bound(const __grid_constant__ CUtensorMap tmap, MatchArgs A, int j0,
                                                        int nj, int nch) {
  begin_after_previous();
  __shared__ __align__(128) float win[MAXCOL * WP];        // staged columns, pitch WP
  __shared__ __align__(16) float nrm[8 * MAXCH * WP];      // per position column: row sums, then -||w16||^2 / 2
  __shared__ __align__(16) __half w16[MAXCOL * HP];        // centred f16 window, pitch HP
  __shared__ __align__(16) uint32_t scratch[NREF][SCR];
  __shared__ uint64_t mbar;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i = blockIdx.x % A.M, jt = j0 + NREF * (int)(blockIdx.x / A.M);
  const int s = A.s, y0 = i * s, o = y0 & 3;  // TMA rows start on a 16-byte boundary; the window o rows later
  if (tid == 0) {
    tc::mbar_init(&mbar, 1);
    tc::fence_mbar_init();
    tc::mbar_expect_tx(&mbar, (8 * nch + 7) * WP * (int)sizeof(float));
    tc::tma_load_2d(win, &tmap, y0 - o, jt * s, &mbar);
  }
  __syncthreads();  // the barrier word is initialised
  bool ok = tc::mbar_wait(&mbar, 0, MATCH_WAIT_CYCLES);
  if (!__syncthreads_and(ok)) {
    // the copy did not land in time: give it the full limit again before the
    // buffer goes away, report, and leave these references' S unwritten
    if (!ok) tc::mbar_wait(&mbar, 0, MATCH_WAIT_CYCLES);
    if (tid == 0 && A.err) atomicOr(A.err, 4);
    return;
  }

  // ---- centre: the mean of 32 pixels around the references (any value keeps
  // the bound valid; every warp makes the same one)
  float m0 = win[o + H + (lane & 7) + (H + (lane >> 3) * (s + 1)) * WP];
#pragma unroll
  for (int q = 16; q >= 1; q >>= 1) m0 += __shfl_xor_sync(0xffffffffu, m0, q);
  m0 *= 1.f / 32.f;

  // ---- rounded window and row sums of squares: thread = (window row, run of
  // chunks); 39 rows x 3 runs.  A chunk makes 8 positions' sums over 8 columns
  // from 8 new columns and the 7 before them.
  const int row = tid % WD, seg = tid / WD;
  bool big = false;
  if (seg < 3) {
    const int c0 = (nch * seg) / 3, c1 = (nch * (seg + 1)) / 3;
    float q[15];
    __half2 hmax = __float2half2_rn(0.f);
    auto load2 = [&](int col, float& q0, float& q1) {
      const __half2 h = __floats2half2_rn(win[o + row + col * WP] - m0, win[o + row + (col + 1) * WP] - m0);
      hmax = __hmax2_nan(hmax, __habs2(h));
      w16[col * HP + row] = __low2half(h);
      w16[(col + 1) * HP + row] = __high2half(h);
      const float2 f = __half22float2(h);
      q0 = f.x * f.x;
      q1 = f.y * f.y;
    };
    // the run's first 7 columns (an 8th value is the next chunk's first and is made again)
    {
      float dummy;
      load2(8 * c0, q[0], q[1]);
      load2(8 * c0 + 2, q[2], q[3]);
      load2(8 * c0 + 4, q[4], q[5]);
      load2(8 * c0 + 6, q[6], dummy);
    }
#pragma unroll 1
    for (int ch = c0; ch < c1; ++ch) {
      const int col = 8 * ch + 7;
#pragma unroll
      for (int u = 0; u < 8; u += 2) load2(col + u, q[7 + u], q[8 + u]);
      float p2[14], p4[12];
#pragma unroll
      for (int u = 0; u < 14; ++u) p2[u] = q[u] + q[u + 1];
#pragma unroll
      for (int u = 0; u < 12; ++u) p4[u] = p2[u] + p2[u + 2];
#pragma unroll
      for (int u = 0; u < 8; ++u) nrm[(8 * ch + u) * WP + row] = p4[u] + p4[u + 4];
#pragma unroll
      for (int u = 0; u < 7; ++u) q[u] = q[u + 8];
    }
    const float2 f = __half22float2(hmax);
    big = !(f.x < 60000.f && f.y < 60000.f);  // an f16 overflow (or NaN): search exhaustively
  }
  // window row 39: read by the MMAs, multiplied by zeros
  for (int col = tid; col < 8 * nch + 7; col += 128) w16[col * HP + WD] = __float2half(0.f);
  big = __syncthreads_or(big);

  // ---- column sums of 8 rows, in place: thread = (position column, half of
  // the 32 rows); both halves of a column belong to one warp
  {
    const int col = 16 * warp + (lane & 15), half = lane >> 4;
    const bool on = col < 8 * nch;
    float4* p = reinterpret_cast<float4*>(nrm + col * WP + 16 * half);
    float v[24], p2[22], p4[20];
    if (on) {
#pragma unroll
      for (int u = 0; u < 6; ++u) {
        const float4 f = p[u];
        v[4 * u] = f.x; v[4 * u + 1] = f.y; v[4 * u + 2] = f.z; v[4 * u + 3] = f.w;
      }
#pragma unroll
      for (int u = 0; u < 22; ++u) p2[u] = v[u] + v[u + 1];
#pragma unroll
      for (int u = 0; u < 20; ++u) p4[u] = p2[u] + p2[u + 2];
    }
    __syncwarp();
    if (on) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        p[u] = make_float4(-0.5f * (p4[4 * u] + p4[4 * u + 4]), -0.5f * (p4[4 * u + 1] + p4[4 * u + 5]),
                           -0.5f * (p4[4 * u + 2] + p4[4 * u + 6]), -0.5f * (p4[4 * u + 3] + p4[4 * u + 7]));
    }
  }
  __syncthreads();

  const int j = jt + warp;
  if (j >= j0 + nj) return;  // past the range (no barrier follows)
  const int g = i + A.M * j, cb = warp * s;  // the reference's first column in the union
  const float* wv = win + o + cb * WP;
  uint32_t* scr = scratch[warp];
  const int K = A.K;
  const unsigned FULL = 0xffffffffu;
  bool listed = false;
  if (!big) {
    // ---- v = <x16, w16> - ||w16||^2 / 2 at every offset.  Lane (gq = lane / 4,
    // t = lane % 4); B's column n stands for candidate row pi(n) = n / 2 + 4 (n & 1) of its
    // block of 8, so that a lane's start values fall on distinct banks.
    const int gq = lane >> 2, t = lane & 3, pig = (gq >> 1) + 4 * (gq & 1);
    float acc[2][4][4];
    const float* np = nrm + (cb + gq) * WP + t;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[mt][nt][e] = np[(16 * mt + 8 * (e >> 1)) * WP + 8 * nt + 4 * (e & 1)];
    // B(k, n) = x(k - pi(n)): of a lane's k = 2t and 2t + 8 (and the odd pair)
    // exactly one is inside the block, so one pair of values and a mask do
    const int r0 = 2 * t - pig, r1 = r0 + 1;
    const uint32_t mlo = (r0 >= 0 ? 0xffffu : 0u) | (r1 >= 0 ? 0xffff0000u : 0u);
    const unsigned short* xs = reinterpret_cast<const unsigned short*>(w16) + (cb + H) * HP + H;
    const unsigned short* x0 = xs + (r0 & 7);
    const unsigned short* x1 = xs + (r1 & 7);
    // A by ldmatrix: matrix (8 candidate columns, 8 window rows); lane l addresses row l % 8 of matrix l / 8
    const uint32_t a16 = tc::smem_u32(w16) + (uint32_t)(cb * HP * 2);
    const uint32_t adr = a16 + (uint32_t)(((lane & 7) + 8 * ((lane >> 3) & 1)) * HP * 2 + (lane >> 4) * 16);
    const uint32_t adr4 = a16 + (uint32_t)(lane * HP * 2 + 4 * 16);
#pragma unroll
    for (int c = 0; c < D; ++c) {
      const uint32_t b = (uint32_t)x0[c * HP] | ((uint32_t)x1[c * HP] << 16);
      const uint32_t b0 = b & mlo, b1 = b & ~mlo;
      uint32_t last[4];  // window rows 32 .. 39 of the four blocks of 8 candidate columns
      ldsm4(last, adr4 + c * HP * 2);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        uint32_t lo[4], hi[4];  // rows 0..15 and 16..31: {b 0..7, b 8..15} x {first 8 rows, next 8}
        ldsm4(lo, adr + (16 * mt + c) * HP * 2);
        ldsm4(hi, adr + (16 * mt + c) * HP * 2 + 32);
        mma_f16(acc[mt][0], lo[0], lo[1], lo[2], lo[3], b0, b1);
        mma_f16(acc[mt][1], lo[2], lo[3], hi[0], hi[1], b0, b1);
        mma_f16(acc[mt][2], hi[0], hi[1], hi[2], hi[3], b0, b1);
        mma_f16(acc[mt][3], hi[2], hi[3], last[2 * mt], last[2 * mt + 1], b0, b1);
      }
    }

    // ---- threshold: the K-th best lane maximum, then theta; when the list
    // would overflow, the K-th best of the lanes' two best
    const float nx = -2.f * nrm[(cb + H) * WP + H];
    float m1 = acc[0][0][0];
#pragma unroll
    for (int e = 1; e < 32; ++e) m1 = fmaxf(m1, acc[e >> 4][(e >> 2) & 3][e & 3]);
    const float v1 = sort_desc(m1, lane);
    float th = 0.5f * (nx - candidate_threshold<Bound8>(nx - 2.f * __shfl_sync(FULL, v1, K - 1), nx));
    uint32_t hits = 0;
#pragma unroll
    for (int e = 0; e < 32; ++e) hits |= acc[e >> 4][(e >> 2) & 3][e & 3] >= th ? 1u << e : 0u;
    int C = __reduce_add_sync(FULL, __popc(hits));
    if (C > 32) {
      float m2 = -3.4e38f;
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        const float v = acc[e >> 4][(e >> 2) & 3][e & 3];
        if (v < m1) m2 = fmaxf(m2, v);
      }
      // the K-th largest of {v1} and {v2}: the largest min(v1[i - 1], v2[K - 1 - i]) over i = 0 .. K
      // (a second best equal to the best is dropped from v2, which only lowers the bound)
      const float v2 = sort_desc(m2, lane);
      const float prev = __shfl_sync(FULL, v1, (lane + 31) & 31), pair = __shfl_sync(FULL, v2, (K - 1 - lane) & 31);
      float best = lane <= K - 1 ? (lane == 0 ? pair : fminf(prev, pair)) : -3.4e38f;
#pragma unroll
      for (int q = 16; q >= 1; q >>= 1) best = fmaxf(best, __shfl_xor_sync(FULL, best, q));
      best = fmaxf(best, __shfl_sync(FULL, v1, K - 1));
      th = 0.5f * (nx - candidate_threshold<Bound8>(nx - 2.f * best, nx));
      hits = 0;
#pragma unroll
      for (int e = 0; e < 32; ++e) hits |= acc[e >> 4][(e >> 2) & 3][e & 3] >= th ? 1u << e : 0u;
      C = __reduce_add_sync(FULL, __popc(hits));
    }
    if (C == D2 * D2 && one_value(wv, lane)) {
      // every distance is exactly zero and the lowest indices win: column 0's first K rows
      hits = 0;
#pragma unroll
      for (int e = 0; e < 16; ++e)
        if (!(e & 2) && gq == 0 && 8 * (e >> 2) + 4 * (e & 1) + t < K) hits |= 1u << e;
      C = K;
    }
    if (C >= K && C <= LCAND) {
      listed = true;
      float* xrow = reinterpret_cast<float*>(scr);
      uint32_t* lS = scr + 64;
      uint2* list = reinterpret_cast<uint2*>(scr + 96);  // (key, window index)
      // the reference block, row-major
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int e = lane + 32 * u;
        xrow[e] = wv[H + (e >> 3) + (H + (e & 7)) * WP];
      }
      int pos = __popc(hits);
#pragma unroll
      for (int q = 1; q < 32; q <<= 1) {
        const int v = __shfl_up_sync(FULL, pos, q);
        if (lane >= q) pos += v;
      }
      pos -= __popc(hits);
      while (hits) {
        const int e = __ffs(hits) - 1;
        hits &= hits - 1;
        const int b = 16 * (e >> 4) + 8 * ((e >> 1) & 1) + gq, a = 8 * ((e >> 2) & 3) + 4 * (e & 1) + t;
        list[pos++].y = (uint32_t)(a + b * D2);
      }
      __syncwarp();
      // ---- exact SSD of the listed candidates, one per lane, in the
      // exhaustive matcher's operation order
      for (int q = lane; q < C; q += 32) {
        const int ix = (int)list[q].y;
        const float* wc = wv + (ix & 31) + (ix >> 5) * WP;
        float d = 0.f;
#pragma unroll
        for (int r = 0; r < D; ++r) {
          const float4 xa = reinterpret_cast<const float4*>(xrow)[2 * r];
          const float4 xb = reinterpret_cast<const float4*>(xrow)[2 * r + 1];
          const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
          for (int c = 0; c < D; ++c) {
            const float e = x[c] - wc[r + c * WP];
            d = fmaf(e, e, d);
          }
        }
        list[q].x = __float_as_uint(d);
      }
      __syncwarp();
      // ---- rank by (distance, index); S(1) is the reference
      for (int q = lane; q < C; q += 32) {
        const uint2 me = list[q];
        const unsigned long long mk = ((unsigned long long)me.x << 32) | me.y;
        int rank = 0;
#pragma unroll 4
        for (int p = 0; p < C; ++p) {
          const uint2 ot = list[p];
          rank += (((unsigned long long)ot.x << 32) | ot.y) < mk ? 1 : 0;
        }
        if (rank < K) lS[rank] = rank == 0 ? (uint32_t)(H + H * D2 + 1) : me.y + 1;
      }
      __syncwarp();
    }
  }
  int count = K;
  if (!listed) count = search_exhaustive<D, D2>(A, wv, scr, lane);
  emit_group<D, D2>(A, g, i, j, wv, scr + 64, count, lane);
}

}  // namespace

bool match_bound_supported(int d, int d2, const MatchArgs& A) {
  return d == D && d2 == D2 && A.s >= 1 && A.s <= D && !A.tol_branch && A.K >= 1 && A.K <= 32;
}

cudaError_t launch_match_bound(const MatchArgs& A, cudaStream_t st) {
  if (A.gn < 0) return cudaSuccess;  // an empty window
  const int nch = (3 * A.s + D2 + 7) / 8;
  CUtensorMap tm;
  if (!encode_search_map(&tm, A.pad, A.R, A.Q, A.P, WP, 8 * nch + 7)) return cudaErrorInvalidValue;
  // the group columns: all, or the strip form's circular window as one or two ranges
  const int lo = A.gn > 0 ? A.g0 / A.M : 0, len = A.gn > 0 ? A.gn / A.M : A.N;
  const int first = len < A.N - lo ? len : A.N - lo;
  const int from[2] = {lo, 0}, count[2] = {first, len - first};
  for (int q = 0; q < 2; ++q) {
    if (count[q] <= 0) continue;
    launch_next(k_match_bound, A.M * ((count[q] + NREF - 1) / NREF), 128, 0, st, tm, A, from[q], count[q], nch);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace gbm3d

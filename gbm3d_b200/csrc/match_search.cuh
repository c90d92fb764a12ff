// Device code shared by the block matchers (match.cu, match_bound.cu): the
// geometry of a staged search window, the exhaustive search of one reference
// by one warp, and the write of a group's S and gathers.
#pragma once
#include "common.cuh"
#include "kernels.cuh"
#include "tc.cuh"

namespace gbm3d {

// Column pitch of a staged search window of WD rows: its first row sits up to
// 3 rows into a TMA box that starts on a 16-byte boundary.
__host__ __device__ constexpr int win_pitch(int wd) { return (wd + 3 + 3) & ~3; }
// Floats of one warp's window buffer (a multiple of 32: 128-byte aligned buffers).
__host__ __device__ constexpr int win_floats(int wd) { return (win_pitch(wd) * wd + 31) & ~31; }
constexpr long long MATCH_WAIT_CYCLES = 4000000000LL;  // ~2 s at 2 GHz

// Exact SSD of the lane's candidates a = lane (a < D2), b = b0 .. b0 + NB - 1: wv is the
// reference's window (row 0, column 0; column pitch win_pitch) in shared memory.
// Candidate b sees t = x(r, c) - y, acc = fmaf(t, t, acc) in (r, c) order (c = xw - b
// ascends with the window column xw).
template <int D, int D2, int NB>
__device__ __forceinline__ void exact_ssd(const float* wv, const int lane, const int b0, float (&acc)[NB]) {
  constexpr int WP = win_pitch(D + D2 - 1);
  constexpr int H = D2 / 2;
#pragma unroll
  for (int b = 0; b < NB; ++b) acc[b] = 0.f;
  const int a = lane < D2 ? lane : 0;
#pragma unroll 1
  for (int r = 0; r < D; ++r) {
    float xr[D];
#pragma unroll
    for (int c = 0; c < D; ++c) xr[c] = wv[(H + r) + (H + c) * WP];
    const float* wrow = wv + (a + r) + b0 * WP;
#pragma unroll
    for (int xw = 0; xw < D + NB - 1; ++xw) {
      const float w = wrow[xw * WP];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int c = xw - b;
        if (c >= 0 && c < D) {
          const float t = xr[c] - w;
          acc[b] = fmaf(t, t, acc[b]);
        }
      }
    }
  }
}

// Selection of a reference's group by one warp from its exact distances: lane a
// holds the candidates (a, b), b = 0 .. D2-1.  lst: 224 words (keys, indices, S and the bounded set).
// Leaves the group's 1-based window indices in lst[64 ..] and returns their count.
template <int D, int D2>
__device__ __forceinline__ int select_group(const MatchArgs& A, const float* wv, const float (&acc)[D2], uint32_t* lst,
                                            const int lane) {
  constexpr int WP = win_pitch(D + D2 - 1);
  constexpr int H = D2 / 2;
  const int a = lane < D2 ? lane : 0;
  // ---- selection -------------------------------------------------------------
  const unsigned FULL = 0xffffffffu;
  uint32_t key[D2];
#pragma unroll
  for (int b = 0; b < D2; ++b) key[b] = lane < D2 ? __float_as_uint(acc[b]) : 0xffffffffu;
  const int K = A.K;
  uint32_t selmask = 0;
  int count = K;
  bool index_order = false;  // tolerance branch with numMin <= #found <= numMax
  int want = K;
  if (A.tol_branch) {
    // matchBlocksCPU.m:89-99: D = ssd/||xR||^2 compared with tol.
    float nR = 0.f;
    for (int c = 0; c < D; ++c)
      for (int r = 0; r < D; ++r) {
        const float xv = wv[(H + r) + (H + c) * WP];
        nR = fmaf(xv, xv, nR);
      }
    int nf = 0;
#pragma unroll
    for (int b = 0; b < D2; ++b)
      if (lane < D2 && __uint_as_float(key[b]) / nR < A.tol) { selmask |= 1u << b; ++nf; }
    const int found = __reduce_add_sync(FULL, nf);
    if (found > K) { want = K; selmask = 0; }
    else if (found < A.numMin) { want = A.numMin; selmask = 0; }
    else { index_order = true; count = found; }
    if (!index_order) count = want;
  }
  // Fast exact path: T = the want-th smallest of the 32 lane minima is >= the
  // want-th smallest key, so the selection lies in {key <= T}.  When that set
  // holds at most 64 keys, rank them by (key, index) directly.
  uint32_t* lkey = lst;
  uint32_t* lidx = lst + 32;
  uint32_t* lS = lst + 64;
  uint32_t* bkey = lst + 96;   // 64 keys and 64 indices of the bounded candidate set
  uint32_t* bidx = lst + 160;
  bool ranked = false;
  if (!index_order) {
    uint32_t lm = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < D2; ++b) lm = min(lm, key[b]);
    // bitonic sort of the lane minima across the warp (ascending by lane)
    uint32_t v = lm;
#pragma unroll
    for (int k2 = 2; k2 <= 32; k2 <<= 1)
#pragma unroll
      for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
        const uint32_t o = __shfl_xor_sync(FULL, v, j2);
        const bool up = ((lane & k2) == 0), lower = ((lane & j2) == 0);
        v = (lower == up) ? min(v, o) : max(v, o);
      }
    uint32_t T = __shfl_sync(FULL, v, want - 1);
    int cl = 0;
#pragma unroll
    for (int b = 0; b < D2; ++b) cl += key[b] <= T ? 1 : 0;
    int C = __reduce_add_sync(FULL, cl);
    if (T != 0xffffffffu && C > 64) {
      // Tighter bound (smooth images, where many keys tie with the lane
      // minima): T2 = the want-th smallest of the 64 values {lane minimum,
      // lane second minimum}, still >= the want-th smallest key.  With A the
      // sorted minima and B the sorted second minima, the want-th smallest of
      // A u B is the smallest max(A[i-1], B[want-1-i]) over i = 0..want.
      uint32_t m1 = 0xffffffffu, m2 = 0xffffffffu;
#pragma unroll
      for (int b = 0; b < D2; ++b) {
        const uint32_t kb = key[b];
        if (kb < m1) { m2 = m1; m1 = kb; } else if (kb < m2) m2 = kb;
      }
      uint32_t vb = m2;
#pragma unroll
      for (int k2 = 2; k2 <= 32; k2 <<= 1)
#pragma unroll
        for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
          const uint32_t o = __shfl_xor_sync(FULL, vb, j2);
          const bool up = ((lane & k2) == 0), lower = ((lane & j2) == 0);
          vb = (lower == up) ? min(vb, o) : max(vb, o);
        }
      const uint32_t a_prev = __shfl_sync(FULL, v, (lane + 31) & 31);          // A[lane - 1]
      const uint32_t b_pair = __shfl_sync(FULL, vb, (want - 1 - lane) & 31);  // B[want - 1 - lane]
      uint32_t cand = 0xffffffffu;
      if (lane <= want - 1)  // i = lane in 0 .. want - 1 (i = want is T itself)
        cand = max(lane == 0 ? 0u : a_prev, b_pair);
      T = min(T, __reduce_min_sync(FULL, cand));
      cl = 0;
#pragma unroll
      for (int b = 0; b < D2; ++b) cl += key[b] <= T ? 1 : 0;
      C = __reduce_add_sync(FULL, cl);
    }
    if (T != 0xffffffffu && C <= 64) {
      int pos = cl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, pos, o);
        if (lane >= o) pos += t;
      }
      pos -= cl;
#pragma unroll
      for (int b = 0; b < D2; ++b)
        if (key[b] <= T) {
          bkey[pos] = key[b];
          bidx[pos] = (uint32_t)(a + b * D2);
          ++pos;
        }
      __syncwarp();
      for (int q = lane; q < C; q += 32) {
        const uint32_t kv = bkey[q], ix = bidx[q];
        int rank = 0;
        for (int t = 0; t < C; ++t) {
          const uint32_t k2 = bkey[t], i2 = bidx[t];
          rank += (k2 < kv || (k2 == kv && i2 < ix)) ? 1 : 0;
        }
        if (rank < want) lS[rank] = rank == 0 ? (uint32_t)(H + H * D2 + 1) : ix + 1;
      }
      ranked = true;
    }
  }
  if (!index_order && !ranked) {
    // radix search for v* = the want-th smallest key (keys are >= +0 floats)
    uint32_t p = 0;
#pragma unroll 1
    for (int bit = 30; bit >= 0; --bit) {
      const uint32_t t = p | ((1u << bit) - 1u);
      int c = 0;
#pragma unroll
      for (int b = 0; b < D2; ++b) c += key[b] <= t ? 1 : 0;
      if (__reduce_add_sync(FULL, c) < want) p |= 1u << bit;
    }
    int lt = 0;
#pragma unroll
    for (int b = 0; b < D2; ++b)
      if (key[b] < p) { selmask |= 1u << b; ++lt; }
    const int need = want - __reduce_add_sync(FULL, lt);
    // ties at v*: lowest column-major index first (b major, a = lane minor)
    int taken = 0;
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int b = 0; b < D2; ++b) {
      const unsigned eq = __ballot_sync(FULL, key[b] == p);
      if (taken < need && eq) {
        const bool mine = (eq >> lane) & 1u;
        if (mine && taken + __popc(eq & below) < need) selmask |= 1u << b;
        taken += __popc(eq);
      }
    }
  }

  // ---- order the selection and write S ---------------------------------------
  if (!ranked) {
  int mine = __popc(selmask);
  int pos = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(FULL, pos, o);
    if (lane >= o) pos += v;
  }
  pos -= mine;
#pragma unroll
  for (int b = 0; b < D2; ++b)
    if ((selmask >> b) & 1u) {
      lkey[pos] = key[b];
      lidx[pos] = (uint32_t)(a + b * D2);
      ++pos;
    }
  __syncwarp();
  const uint32_t ref_idx = (uint32_t)(H + H * D2 + 1);  // matchBlocksCPU.m:103
  if (lane < count) {
    const uint32_t kv = lkey[lane], ix = lidx[lane];
    int rank = 0;
    for (int t = 0; t < count; ++t) {
      const uint32_t k2 = lkey[t], i2 = lidx[t];
      if (index_order) rank += i2 < ix ? 1 : 0;
      else rank += (k2 < kv || (k2 == kv && i2 < ix)) ? 1 : 0;
    }
    lS[rank] = rank == 0 ? ref_idx : ix + 1;
  }
  }
  __syncwarp();
  return count;
}

// The exhaustive search of one reference by one warp.
template <int D, int D2>
__device__ __forceinline__ int search_exhaustive(const MatchArgs& A, const float* wv, uint32_t* lst, const int lane) {
  float acc[D2];
  exact_ssd<D, D2, D2>(wv, lane, 0, acc);
  return select_group<D, D2>(A, wv, acc, lst, lane);
}

// Write the group's S and count, and the optional gathers.
template <int D, int D2>
__device__ __forceinline__ void emit_group(const MatchArgs& A, const int g, const int i, const int j, const float* wv,
                                           const uint32_t* lS, const int count, const int lane) {
  constexpr int WP = win_pitch(D + D2 - 1);
  constexpr int H = D2 / 2;
  const int K = A.K;
  uint32_t* Sg = A.S + (size_t)g * K;
  if (lane < K) Sg[lane] = lane < count ? lS[lane] : 0u;
  if (lane == 0 && A.cnt) A.cnt[g] = count;

  // ---- optional gathers: Volume (matchBlocksCPU.m:107-114), V1/V2 (matchBlocksWie.m:85-89)
  if (A.volume) {
    const size_t mn = (size_t)A.m * A.n;
    float* vol0 = A.volume + (size_t)(i * D) + (size_t)A.m * (j * D);
    if (D == 8 && (A.m & 3) == 0 && (reinterpret_cast<uintptr_t>(A.volume) & 15) == 0) {
      // two slots per pass: lane = (slot parity, column c, half-column r0); each
      // lane stores four rows of one column as one 16-byte store (a block
      // column is 32 contiguous bytes of the volume, 16-byte aligned here).
      // The window pitch is a multiple of 4, so the eight columns of one half
      // take every fourth bank: each lane reads its four rows in an order
      // rotated by u0, which puts the four (parity, half) sets on the four
      // residues, 32 distinct banks per load instead of three or four lanes on one
      const int q = lane & 15, c = q >> 1, r0 = 4 * (q & 1);
      for (int k = lane >> 4; k < K; k += 2) {
        int aa = H, bb = H;
        if (k < count) {
          const int e = (int)lS[k] - 1;
          if ((unsigned)e < (unsigned)(D2 * D2)) { aa = e % D2; bb = e / D2; }
        }
        const float* ws = wv + aa + r0 + (bb + c) * WP;
        const int u0 = (2 * (q & 1) + (lane >> 4) - (int)(tc::smem_u32(ws) >> 2)) & 3;
        float f[4], h[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) f[t] = ws[(t + u0) & 3];
#pragma unroll
        for (int t = 0; t < 4; ++t) h[t] = u0 & 1 ? f[(t + 3) & 3] : f[t];
        *reinterpret_cast<float4*>(vol0 + r0 + (size_t)A.m * c + mn * k) =
            u0 & 2 ? make_float4(h[2], h[3], h[0], h[1]) : make_float4(h[0], h[1], h[2], h[3]);
      }
    } else {
    // lane-parallel over the block: element t = lane + 32 u is row t % D, column t / D
    for (int k = 0; k < K; ++k) {
      int aa = H, bb = H;
      if (k < count) {
        const int e = (int)lS[k] - 1;
        if ((unsigned)e < (unsigned)(D2 * D2)) { aa = e % D2; bb = e / D2; }
      }
      const float* wsrc = wv + aa + bb * WP;
#pragma unroll
      for (int u = 0; u < (D * D + 31) / 32; ++u) {
        const int t = lane + 32 * u;
        if (t < D * D) {
          const int r = t % D, c = t / D;
          vol0[(size_t)r + (size_t)A.m * c + mn * k] = wsrc[r + c * WP];
        }
      }
    }
    }
  }
  if (A.V1 || A.V2) {
    const float* src2 = A.pad2 + (size_t)i * A.s + (size_t)j * A.s * A.P;
    for (int k = 0; k < K; ++k) {
      int e = (int)lS[k] - 1;
      if ((unsigned)e >= (unsigned)(D2 * D2)) e = H + H * D2;
      const int aa = e % D2, bb = e / D2;
      float* o1 = A.V1 ? A.V1 + (size_t)D * D * (k + (size_t)K * g) : nullptr;
      float* o2 = A.V2 ? A.V2 + (size_t)D * D * (k + (size_t)K * g) : nullptr;
      for (int t = lane; t < D * D; t += 32) {
        const int r = t % D, c = t / D;
        if (o1) o1[t] = wv[(aa + r) + (bb + c) * WP];
        if (o2) o2[t] = src2[(aa + r) + (size_t)(bb + c) * A.P];
      }
    }
  }
}

}  // namespace gbm3d

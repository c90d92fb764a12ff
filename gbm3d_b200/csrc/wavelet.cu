// Step 1: global 3D wavelet hard thresholding of the block-group volume.
//
// Restates denoiseAndAggregateGPU.m:27-47 with myWavDec3DFFT.m:10-23 and
// myWavRec3DGPUfast.m:10-40.  The reference filters the whole m x n x K volume
// with circular 3D convolutions through fftn; the filters are outer products
// of 1D factors, so each level here is three separable passes computed
// directly (no FFT), tile by tile in shared memory:
//
//   analysis  : z-pass (slot axis), x-pass, y-pass, each with decimation by 2,
//               c[q] = sum_k h[k] u[(2q - k) mod L]; hard threshold fused into
//               the y-pass store (strict |c| > tau, the approximation kept).
//   synthesis : y-pass, x-pass, z-pass, each upsampling by 2 and correlating,
//               r[p] = sum_band sum_k g[k] up[(p + k) mod L] (lo band first).
//
// Every sum is a serial fmaf chain over nonzero taps in ascending tap index,
// the order the CPU oracle follows.  The cycle spin of the reference
// (circshift of the volume by [s,s,s] before analysis and back after
// synthesis) is folded into the level-1 read and write indices, and the
// average over spins with the clamp max(.,0) is fused into the last level-1
// synthesis pass.
#include "common.cuh"
#include "kernels.cuh"

namespace gbm3d {

// Address parts of a synthesis output: rows (y, z) and columns x, for the two
// layouts of SynthOut.
__device__ __forceinline__ size_t synth_row(const SynthOut& o, int y, int z, int Oy, int Ox, int Oz) {
  if (o.gs == 0) return (size_t)y + (size_t)Oy * Ox * z;
  return ((size_t)((y >> o.gs) * Oz + z) << (2 * o.gs)) + (y & ((1 << o.gs) - 1));
}
__device__ __forceinline__ size_t synth_col_step(const SynthOut& o, int Oy, int Oz) {
  return o.gs == 0 ? (size_t)Oy : (size_t)((Oy >> o.gs) * Oz) << (2 * o.gs);
}
__device__ __forceinline__ size_t synth_col(const SynthOut& o, int x, size_t step) {
  return (size_t)(x >> o.gs) * step + (size_t)((x & ((1 << o.gs) - 1)) << o.gs);
}

constexpr int TQ = 32;  // analysis output tile (coefficients per axis)
constexpr int TP = 32;  // synthesis output tile (samples per axis)

__global__ void __launch_bounds__(256) k_wav_analysis(const float* __restrict__ in, int Ly, int Lx,
                                                      int Lz, int shift, float* __restrict__ out,
                                                      WaveletBank bk, LevelBands th, int tx0) {
  extern __shared__ float sm[];
  const int R = bk.reach_a;
  const int NY = 2 * TQ + R;
  float* tz = sm;                // [2][NY(x)][NY(y)]
  float* tx = sm + 2 * NY * NY;  // [4][TQ(qx)][NY(y)]
  const int Oy = Ly >> 1, Ox = Lx >> 1, Oz = Lz >> 1;
  const int ntx = (Ox + TQ - 1) / TQ, bx = blockIdx.y + tx0;  // column tile: the window's, modulo the count
  const int qy0 = blockIdx.x * TQ, qx0 = (bx >= ntx ? bx - ntx : bx) * TQ, qz = blockIdx.z;
  const int y0 = 2 * qy0 - R, x0 = 2 * qx0 - R;
  const size_t plane = (size_t)Ly * Lx;

  // load + z-pass (slot axis)
  for (int e = threadIdx.x; e < NY * NY; e += blockDim.x) {
    const int yy = e % NY, xx = e / NY;
    const int y = pmod(y0 + yy - shift, Ly), x = pmod(x0 + xx - shift, Lx);
    const float* col = in + y + (size_t)Ly * x;
#pragma unroll
    for (int fz = 0; fz < 2; ++fz) {
      const Taps& t = bk.z.a[fz];
      float acc = 0.f;
      for (int u = 0; u < t.n; ++u) {
        const int k = t.k[u];
        if (k >= Lz) continue;
        acc = fmaf(t.h[u], col[plane * pmod(2 * qz - k - shift, Lz)], acc);
      }
      tz[fz * NY * NY + e] = acc;
    }
  }
  __syncthreads();
  // x-pass
  for (int e = threadIdx.x; e < 4 * TQ * NY; e += blockDim.x) {
    const int yy = e % NY, qx = (e / NY) % TQ, comb = e / (NY * TQ);
    const int fx = comb & 1, fz = comb >> 1;
    const float* src = tz + fz * NY * NY + yy;
    const Taps& t = bk.xy.a[fx];
    float acc = 0.f;
    for (int u = 0; u < t.n; ++u) {
      const int k = t.k[u];
      if (k >= Lx) continue;
      acc = fmaf(t.h[u], src[(2 * qx + R - k) * NY], acc);
    }
    tx[(comb * TQ + qx) * NY + yy] = acc;
  }
  __syncthreads();
  // y-pass + hard threshold + store
  const size_t bsz = (size_t)Oy * Ox * Oz;
  for (int e = threadIdx.x; e < 8 * TQ * TQ; e += blockDim.x) {
    const int qy = e % TQ, qx = (e / TQ) % TQ, code = e / (TQ * TQ);
    if (qy0 + qy >= Oy || qx0 + qx >= Ox) continue;
    const int fy = code & 1, comb = code >> 1;
    const float* src = tx + (comb * TQ + qx) * NY;
    const Taps& t = bk.xy.a[fy];
    float acc = 0.f;
    for (int u = 0; u < t.n; ++u) {
      const int k = t.k[u];
      if (k >= Ly) continue;
      acc = fmaf(t.h[u], src[2 * qy + R - k], acc);
    }
    if (code) acc = acc * (fabsf(acc) > th.tau[code] ? 1.f : 0.f);
    out[code * bsz + (qy0 + qy) + (size_t)Oy * ((qx0 + qx) + (size_t)Ox * qz)] = acc;
  }
}

__global__ void __launch_bounds__(256) k_wav_synthesis(const float* __restrict__ bands,
                                                       const float* __restrict__ approx, int Oy,
                                                       int Ox, int Oz, SynthOut o, WaveletBank bk, int tx0) {
  extern __shared__ float sm[];
  const int Iy = Oy >> 1, Ix = Ox >> 1, Iz = Oz >> 1;
  const int NQ = (TP - 1 + bk.reach_s) / 2 + 1;
  float* B = sm;                  // [8][NQ(qx)][NQ(qy)]
  float* Y = B + 8 * NQ * NQ;     // [4][NQ(qx)][TP(py)]
  float* X = Y + 4 * NQ * TP;     // [2][TP(px)][TP(py)]
  const int ntx = (Ox + TP - 1) / TP, bx = blockIdx.y + tx0;
  const int py0 = blockIdx.x * TP, px0 = (bx >= ntx ? bx - ntx : bx) * TP, qz = blockIdx.z;
  const int qy0 = py0 >> 1, qx0 = px0 >> 1;
  const size_t bsz = (size_t)Iy * Ix * Iz;

  for (int e = threadIdx.x; e < 8 * NQ * NQ; e += blockDim.x) {
    const int qyl = e % NQ, qxl = (e / NQ) % NQ, code = e / (NQ * NQ);
    const int qy = (qy0 + qyl) % Iy, qx = (qx0 + qxl) % Ix;
    const float* src = code ? bands + code * bsz : approx;
    B[e] = src[qy + (size_t)Iy * (qx + (size_t)Ix * qz)];
  }
  __syncthreads();
  // y-pass: combine fy for each (fx, fz)
  for (int e = threadIdx.x; e < 4 * NQ * TP; e += blockDim.x) {
    const int py = e % TP, qxl = (e / TP) % NQ, comb = e / (TP * NQ);
    float acc = 0.f;
#pragma unroll
    for (int fy = 0; fy < 2; ++fy) {
      const float* src = B + (fy + 2 * comb) * NQ * NQ + qxl * NQ;
      const Taps& t = bk.xy.s[fy];
      for (int u = 0; u < t.n; ++u) {
        const int k = t.k[u];
        if (k >= Oy || ((py + k) & 1)) continue;
        acc = fmaf(t.h[u], src[(py + k) >> 1], acc);
      }
    }
    Y[(comb * NQ + qxl) * TP + py] = acc;
  }
  __syncthreads();
  // x-pass: combine fx for each fz
  for (int e = threadIdx.x; e < 2 * TP * TP; e += blockDim.x) {
    const int py = e % TP, px = (e / TP) % TP, fz = e / (TP * TP);
    float acc = 0.f;
#pragma unroll
    for (int fx = 0; fx < 2; ++fx) {
      const float* src = Y + (fx + 2 * fz) * NQ * TP + py;
      const Taps& t = bk.xy.s[fx];
      for (int u = 0; u < t.n; ++u) {
        const int k = t.k[u];
        if (k >= Ox || ((px + k) & 1)) continue;
        acc = fmaf(t.h[u], src[((px + k) >> 1) * TP], acc);
      }
    }
    X[(fz * TP + px) * TP + py] = acc;
  }
  __syncthreads();
  // z-pass: outputs pz = 2qz (tap 0) and pz = 2qz-1 (tap 1); write / accumulate
  for (int e = threadIdx.x; e < 2 * TP * TP; e += blockDim.x) {
    const int py = e % TP, px = (e / TP) % TP, which = e / (TP * TP);
    if (py0 + py >= Oy || px0 + px >= Ox) continue;
    const int pz = pmod(2 * qz - which, Oz);
    float acc = 0.f;
#pragma unroll
    for (int fz = 0; fz < 2; ++fz) {
      const Taps& t = bk.z.s[fz];
      for (int u = 0; u < t.n; ++u) {
        const int k = t.k[u];
        if (k >= Oz || k != which) continue;
        acc = fmaf(t.h[u], X[(fz * TP + px) * TP + py], acc);
      }
    }
    const int oy = pmod(py0 + py - o.shift, Oy), ox = pmod(px0 + px - o.shift, Ox), oz = pmod(pz - o.shift, Oz);
    float* dst = o.out + synth_row(o, oy, oz, Oy, Ox, Oz) + synth_col(o, ox, synth_col_step(o, Oy, Oz));
    float v = o.first ? acc : *dst + acc;
    if (o.last) {
      v = v / o.cycles;
      v = v > 0.f ? v : 0.f;
      if (o.clamp1) v = fminf(v, 1.f);
    }
    *dst = v;
  }
}

// getBM3DAggWeights(3,1) (getBM3DAggWeights.m:11-19) and weight = 1/(D+eps)
// (denoiseAndAggregateGPU.m:75), one warp per group.  Each of the three sums
// is a fixed-order reduction: lane l adds the elements l, l+32, ... of the
// column-major difference array in order, then an xor butterfly.
__device__ __forceinline__ float d3(float u0, float u1, float u2, float u3) {
  const float a0 = u1 - u0, a1 = u2 - u1, a2 = u3 - u2;
  const float b0 = a1 - a0, b1 = a2 - a1;
  return b1 - b0;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

__global__ void __launch_bounds__(128) k_ht_weights(const float* __restrict__ V, int m, int n, int M,
                                                    int N, int d, int K, const int32_t* __restrict__ cnt,
                                                    float* __restrict__ wgt, int g0, int gn) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = window_group(blockIdx.x * 4 + warp, g0, gn, M * N);
  if (g < 0) return;
  const int i = g % M, j = g / M;
  const int nm = cnt ? cnt[g] : K;
  const size_t sz = (size_t)m * n;
  const float* base = V + (size_t)i * d + (size_t)j * d * m;
  auto at = [&](int r, int c, int k) { return base[r + (size_t)c * m + sz * k]; };
  const int dm = d - 3;
  float tx = 0.f, ty = 0.f, tz = 0.f;
  const int nx = d * dm * nm;
  for (int e = lane; e < nx; e += 32) {
    const int r = e % d, c = (e / d) % dm, k = e / (d * dm);
    tx = tx + fabsf(d3(at(r, c, k), at(r, c + 1, k), at(r, c + 2, k), at(r, c + 3, k)));
  }
  for (int e = lane; e < nx; e += 32) {
    const int r = e % dm, c = (e / dm) % d, k = e / (dm * d);
    ty = ty + fabsf(d3(at(r, c, k), at(r + 1, c, k), at(r + 2, c, k), at(r + 3, c, k)));
  }
  const int nzz = d * d * (nm - 1);
  for (int e = lane; e < nzz; e += 32) {
    const int r = e % d, c = (e / d) % d, k = e / (d * d);
    tz = tz + fabsf(at(r, c, k + 1) - at(r, c, k));
  }
  tx = warp_sum(tx);
  ty = warp_sum(ty);
  tz = warp_sum(tz);
  if (lane == 0) {
    float w = tx * 0.25f + ty * 0.25f;
    w = w + tz;
    wgt[g] = 1.f / (w + 2.220446049250313e-16f);
  }
}

// ---------------------------------------------------------------------------
// The three separable banks of the pipelines, with tap positions known at
// compile time:
//   analysis  lo: taps 0 .. LL-1      hi: taps H0 .. H0+HN-1
//   synthesis lo: taps S0 .. S0+SN-1  hi: taps 0 .. SH-1
//   slot axis: taps 0, 1 for all four filters
// (bior1.5 x Haar LL = SH = 10, H0 = S0 = 4, HN = SN = 2; 3D Haar all 2 from 0;
// sym4 x Haar, VBM3D's bank, all 8 from 0).
//
// One warp marches along the slow axis x over a strip of the fast axis y, for
// one pair of slots, with the x window in registers; no block barrier.  A
// tile-per-CTA version spent 60-70 % of the issue slots, two thirds of them on
// index arithmetic and on passing every intermediate through shared memory;
// here a value is loaded once, both x inputs of a step come from registers,
// and only the y pass (neighbouring lanes) goes through the warp's own piece
// of shared memory.  Each output is the same serial fmaf chain, over the same taps in
// the same order, as in the generic kernels and the oracle.  Any size of at
// least the filter length works (indices wrap modulo the size once per strip),
// so the small coarse levels run here too.
//   Measured (all launches of a call, analysis / synthesis): 4096^2 tuned 0.80 -> 0.61 /
// 0.92 -> 0.61 ms (the floor of one read and one write per voxel is 0.38),
// dense 21.5 -> 15.4 / 28.2 -> 21.5 ms (floor 10.6 / 13), 128 x 96 with the generic
// coarse levels 559 -> 113 / 398 -> 114 us, VBM3D at 720p (8 frames) 2.45 -> 1.62 /
// 4.29 -> 1.83 ms.  At 1024^2 dense level 0 moves its bytes at 62 % (analysis)
// and 50 % (synthesis) of the copy bandwidth; shared-memory pipe and issue are at 55-65 %
// at 16 warps per SM (register windows).
// ---------------------------------------------------------------------------
struct FastBank {
  float alo[10], ahi[10], slo[10], shi[10];
  float azl[2], azh[2], szl[2], szh[2];
};

constexpr int MW = 4;  // warps per CTA
constexpr long MARCH_WARPS = 148 * 32;  // warps that a launch should have, where its size allows

constexpr int imax(int a, int b) { return a > b ? a : b; }

// Analysis.  Lane l holds two neighbouring rows of coefficient row q = q0 + l - HL: 2q and
// 2q + 1 at an even shift, 2q - 1 and 2q at an odd one, whichever pair starts on 8 bytes in
// memory.  The HL lanes in front are the halo of the y pass, so a warp makes 32 - HL
// rows.  Step t loads columns 2 qx - 1 and 2 qx of both slots PD steps ahead, applies the
// slot pass, then the x pass on the last W columns, and hands the four (fx, fz)
// results to the neighbouring lanes for the y pass, the threshold and the store.
template <int LL, int H0, int HN, bool EVEN>
__global__ void __launch_bounds__(32 * MW, 4) k_wav_analysis_march(const float* __restrict__ in, int Ly, int Lx,
                                                                   int Lz, int shift, float* __restrict__ out,
                                                                   FastBank fb, LevelBands th, int ty, int x_lo,
                                                                   int x_len, int seg, SpinSet sp) {
  begin_after_previous(in);
  constexpr int W = imax(LL, H0 + HN), HX = W / 2 - 1, HL = EVEN ? W / 2 : W / 2 - 1;
  constexpr int U = W > 2 ? W / 2 : 4, PD = 3;
  static_assert(W % 2 == 0 && (2 * U) % W == 0 && PD < U, "the window repeats every U steps");
  __shared__ float2 sb[MW][2][4][32 + HL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int Oy = Ly >> 1, Ox = Lx >> 1, Oz = Lz >> 1;
  const int sgi = blockIdx.y, strip = blockIdx.x * MW + warp;
  if (strip >= ty) return;
  int qz = blockIdx.z;
  if (sp.n > 1) {
    const int spin = qz / Oz;
    qz -= spin * Oz;
    in += spin * sp.in;
    out += spin * sp.out;
  }
  const int q = strip * (32 - HL) - HL + lane;
  const bool live = lane >= HL && q < Oy;
  const size_t plane = (size_t)Ly * Lx;
  // lane offsets stay 32 bits and the rest of every address is the same for the
  // whole CTA (slots, columns, bands), so it lives in uniform registers
  const unsigned yo = pmod(EVEN ? 2 * q - shift : 2 * q - 1 - shift, Ly);
  const float* i0 = in + plane * pmod(2 * qz - shift, Lz);      // slot tap 0
  const float* i1 = in + plane * pmod(2 * qz - 1 - shift, Lz);  // slot tap 1
  const int xs = x_lo + sgi * seg, n = min(seg, x_len - sgi * seg), T = n + HX;
  int xc = pmod(2 * (xs - HX) - 1 - shift, Lx);  // next column to load
  int ox = xs >= Ox ? xs - Ox : xs;
  float* dst = out + (size_t)Oy * Ox * qz;
  const size_t bsz = (size_t)Oy * Ox * Oz;
  float2(*sw)[4][32 + HL] = sb[warp];

  float2 nx[U][4];   // loaded columns: [2 column + slot], the lane's two rows
  float w[2][2][W];  // slot-pass results [fz][row][column], a ring of W columns
  auto load = [&](float2 (&v)[4]) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      v[2 * c] = __ldg(reinterpret_cast<const float2*>(i0 + (size_t)Ly * xc + yo));
      v[2 * c + 1] = __ldg(reinterpret_cast<const float2*>(i1 + (size_t)Ly * xc + yo));
      xc = xc + 1 == Lx ? 0 : xc + 1;
    }
  };
#pragma unroll
  for (int p = 0; p < PD; ++p)
    if (p < T) load(nx[p]);
  for (int t0 = 0; t0 < T; t0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u;
      if (t >= T) break;
      if (t + PD < T) load(nx[(u + PD) % U]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 v0 = nx[u][2 * c], v1 = nx[u][2 * c + 1];
        w[0][0][(2 * u + c) % W] = fmaf(fb.azl[1], v1.x, fmaf(fb.azl[0], v0.x, 0.f));
        w[0][1][(2 * u + c) % W] = fmaf(fb.azl[1], v1.y, fmaf(fb.azl[0], v0.y, 0.f));
        w[1][0][(2 * u + c) % W] = fmaf(fb.azh[1], v1.x, fmaf(fb.azh[0], v0.x, 0.f));
        w[1][1][(2 * u + c) % W] = fmaf(fb.azh[1], v1.y, fmaf(fb.azh[0], v0.y, 0.f));
      }
      if (t >= HX) {
        // x pass: tap k reads column 2 qx - k, the ring's entry 2u + 1 - k
        float2 own[4];
#pragma unroll
        for (int fz = 0; fz < 2; ++fz) {
          float lo[2], hi[2];
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            lo[y] = hi[y] = 0.f;
#pragma unroll
            for (int k = 0; k < LL; ++k) lo[y] = fmaf(fb.alo[k], w[fz][y][(2 * u + 1 - k + W) % W], lo[y]);
#pragma unroll
            for (int k = 0; k < HN; ++k) hi[y] = fmaf(fb.ahi[k], w[fz][y][(2 * u + 1 - H0 - k + W) % W], hi[y]);
          }
          own[2 * fz] = make_float2(lo[0], lo[1]);
          own[2 * fz + 1] = make_float2(hi[0], hi[1]);
        }
        float2(*sp)[32 + HL] = sw[t & 1];  // the two halves alternate, so one barrier per step does
#pragma unroll
        for (int comb = 0; comb < 4; ++comb) sp[comb][lane + HL] = own[comb];
        __syncwarp();
        // y pass: tap k reads row 2q - k
        float* d = dst + (size_t)Oy * ox;
#pragma unroll
        for (int comb = 0; comb < 4; ++comb) {
          const float2* nb = &sp[comb][lane + HL];
          float v[W + 1];
          if (EVEN) {
            v[0] = own[comb].x;
#pragma unroll
            for (int p = 1; p < HL; ++p) {
              const float2 f = nb[-p];
              v[2 * p - 1] = f.y;
              v[2 * p] = f.x;
            }
            v[2 * HL - 1] = nb[-HL].y;
          } else {
            v[0] = own[comb].y;
            v[1] = own[comb].x;
#pragma unroll
            for (int p = 1; p <= HL; ++p) {
              const float2 f = nb[-p];
              v[2 * p] = f.y;
              v[2 * p + 1] = f.x;
            }
          }
          float lo = 0.f, hi = 0.f;
#pragma unroll
          for (int k = 0; k < LL; ++k) lo = fmaf(fb.alo[k], v[k], lo);
#pragma unroll
          for (int k = 0; k < HN; ++k) hi = fmaf(fb.ahi[k], v[H0 + k], hi);
          if (comb) lo = lo * (fabsf(lo) > th.tau[2 * comb] ? 1.f : 0.f);
          hi = hi * (fabsf(hi) > th.tau[2 * comb + 1] ? 1.f : 0.f);
          if (live) {
            (d + (size_t)(2 * comb) * bsz)[(unsigned)q] = lo;
            (d + (size_t)(2 * comb + 1) * bsz)[(unsigned)q] = hi;
          }
        }
        ox = ox + 1 == Ox ? 0 : ox + 1;
      }
    }
  }
}

// Synthesis.  Lane l makes the rows 2q and 2q + 1 of pair q = q0 + l.  Step t has the
// eight bands' coefficients of column t (rows q0 .. q0 + 31 + HS) in a ring of NST
// staged columns (cp.async, NST - 1 columns in flight), applies the y pass for the four (fx, fz)
// and, once HS columns are ahead, the x pass and the slot pass for the column
// pair t - HS from the register windows.
//   RMW adds to the sums of earlier cycle spins; PAIR: an even shift, so the two
// rows are neighbours at an 8-byte boundary.
__device__ __noinline__ float2 divide2(float2 v, float c) { return make_float2(v.x / c, v.y / c); }

template <int S0, int SN, int SH, bool RMW, bool PAIR>
__global__ void __launch_bounds__(32 * MW, 4) k_wav_synthesis_march(const float* __restrict__ bands,
                                                                 const float* __restrict__ approx, int Oy, int Ox,
                                                                 int Oz, SynthOut o, FastBank fb, int ty, int x_lo,
                                                                 int x_len, int seg, SpinSet sp) {
  begin_after_previous(bands, approx);
  constexpr int W = imax(S0 + SN, SH), HS = W / 2, RW = HS + 1, NST = 4, PQ = 40;
  static_assert(W % 2 == 0 && 32 + HS <= PQ && 8 * HS <= 64, "ring");
  __shared__ float ring[MW][NST][8][PQ];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int Iy = Oy >> 1, Ix = Ox >> 1, Iz = Oz >> 1;
  const int sgi = blockIdx.y, strip = blockIdx.x * MW + warp;
  if (strip >= ty) return;
  int qz = blockIdx.z;
  if (sp.n > 1) {
    const int spin = qz / Iz;
    qz -= spin * Iz;
    bands += spin * sp.in;
    approx += spin * sp.approx;
    o.out += spin * sp.out;
  }
  const int q0 = strip * 32, q = q0 + lane;
  const bool live = q < Iy;
  const size_t bsz = (size_t)Iy * Ix * Iz, zoff = (size_t)Iy * Ix * qz;
  const int xs = x_lo + sgi * seg, n = min(seg, x_len - sgi * seg), T = n + HS;
  float(*rb)[8][PQ] = ring[warp];

  // staging: lane's own row of the eight bands, and its share of the HS rows past them
  const float* pa = approx + zoff;
  const float* pb = bands + zoff;
  const unsigned yo = q % Iy;
  const float* ph[2];
  int hd[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int e = lane + 32 * h, code = e / HS, off = 32 + e % HS;
    hd[h] = e < 8 * HS ? code * PQ + off : -1;
    ph[h] = (code && e < 8 * HS ? bands + code * bsz : approx) + zoff + (q0 + off) % Iy;
  }
  int xc = xs >= Ix ? xs - Ix : xs;  // next column to stage
  auto stage = [&](int slot) {
    float* s = &rb[slot][0][0];
    const size_t col = (size_t)Iy * xc;
    cp_async4(s + lane, pa + col + yo);
#pragma unroll
    for (int code = 1; code < 8; ++code) cp_async4(s + code * PQ + lane, pb + code * bsz + col + yo);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (hd[h] >= 0) cp_async4(s + hd[h], ph[h] + col);
    xc = xc + 1 == Ix ? 0 : xc + 1;
  };

  // outputs: rows 2q, 2q + 1 (lane offsets) and slots 2 qz, 2 qz - 1, shifted back
  const unsigned oA = (unsigned)synth_row(o, pmod(2 * q - o.shift, Oy), 0, Oy, Ox, Oz);
  const unsigned oB = (unsigned)synth_row(o, pmod(2 * q + 1 - o.shift, Oy), 0, Oy, Ox, Oz);
  float* const dz[2] = {o.out + synth_row(o, 0, pmod(2 * qz - o.shift, Oz), Oy, Ox, Oz),
                        o.out + synth_row(o, 0, pmod(2 * qz - 1 - o.shift, Oz), Oy, Ox, Oz)};
  const size_t cstep = synth_col_step(o, Oy, Oz);
  const int cmask = (1 << o.gs) - 1;
  int ox = pmod(2 * xs - o.shift, Ox);
  size_t col = synth_col(o, ox, cstep);
  auto after = [&](int x, size_t c) {  // the column after x
    return x + 1 == Ox ? (size_t)0 : (x + 1) & cmask ? c + ((size_t)1 << o.gs) : (size_t)((x + 1) >> o.gs) * cstep;
  };

#pragma unroll
  for (int p = 0; p < NST - 1; ++p) {
    if (p < T) stage(p);
    cp_async_commit();
  }
  // y-pass results [fz][row][column], lo and hi in x; moved down every step
  // (unrolling the six-step ring instead of moving it stalled on instruction fetch)
  float wl[2][2][RW] = {}, wh[2][2][RW] = {};
  for (int t = 0; t < T; ++t) {
    cp_async_wait_group<NST - 2>();
    __syncwarp();  // column t is staged; every lane has left column t - 1
    if (t + NST - 1 < T) stage((t + NST - 1) % NST);
    cp_async_commit();
    // the sums of the earlier cycle spins, in flight over this step's passes
    const size_t cols[2] = {col, after(ox, col)};
    float2 prev[2][2];
    if (RMW && t >= HS && live) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const float* p = dz[z] + cols[c];
          prev[c][z] = PAIR ? *reinterpret_cast<const float2*>(p + oA) : make_float2(p[oA], p[oB]);
        }
    }
    const float* s = &rb[t % NST][0][lane];
#pragma unroll
    for (int comb = 0; comb < 4; ++comb) {
      const float* sl = s + 2 * comb * PQ;
      const float* sh = sl + PQ;
      float cl[HS + 1], ch[HS + 1];
#pragma unroll
      for (int p = 0; p <= HS; ++p) {  // only the entries that taps use are read
        if (p >= S0 / 2 && p <= (S0 + SN) / 2) cl[p] = sl[p];
        if (p <= SH / 2) ch[p] = sh[p];
      }
      float ev = 0.f, od = 0.f;
#pragma unroll
      for (int k = S0; k < S0 + SN; ++k) {
        if (k % 2 == 0) ev = fmaf(fb.slo[k - S0], cl[k / 2], ev);
        else od = fmaf(fb.slo[k - S0], cl[(k + 1) / 2], od);
      }
#pragma unroll
      for (int k = 0; k < SH; ++k) {
        if (k % 2 == 0) ev = fmaf(fb.shi[k], ch[k / 2], ev);
        else od = fmaf(fb.shi[k], ch[(k + 1) / 2], od);
      }
      if (comb & 1) {
        wh[comb >> 1][0][HS] = ev;
        wh[comb >> 1][1][HS] = od;
      } else {
        wl[comb >> 1][0][HS] = ev;
        wl[comb >> 1][1][HS] = od;
      }
    }
    if (t >= HS) {
      // x pass of the column pair j = t - HS: tap k reads column j + ceil(k / 2)
      float xv[2][2][2];  // [fz][row][even, odd column]
#pragma unroll
      for (int fz = 0; fz < 2; ++fz)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          float ev = 0.f, od = 0.f;
#pragma unroll
          for (int k = S0; k < S0 + SN; ++k) {
            if (k % 2 == 0) ev = fmaf(fb.slo[k - S0], wl[fz][y][k / 2], ev);
            else od = fmaf(fb.slo[k - S0], wl[fz][y][(k + 1) / 2], od);
          }
#pragma unroll
          for (int k = 0; k < SH; ++k) {
            if (k % 2 == 0) ev = fmaf(fb.shi[k], wh[fz][y][k / 2], ev);
            else od = fmaf(fb.shi[k], wh[fz][y][(k + 1) / 2], od);
          }
          xv[fz][y][0] = ev;
          xv[fz][y][1] = od;
        }
      // slot pass: slot 2 qz from tap 0, slot 2 qz - 1 from tap 1; write or accumulate
      if (live) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            float2 v = make_float2(fmaf(fb.szh[z], xv[1][0][c], fmaf(fb.szl[z], xv[0][0][c], 0.f)),
                                   fmaf(fb.szh[z], xv[1][1][c], fmaf(fb.szl[z], xv[0][1][c], 0.f)));
            if (RMW) v = make_float2(prev[c][z].x + v.x, prev[c][z].y + v.y);
            if (o.last) {
              v = o.pow2 ? make_float2(v.x * o.inv, v.y * o.inv) : divide2(v, o.cycles);
              v = make_float2(v.x > 0.f ? v.x : 0.f, v.y > 0.f ? v.y : 0.f);
              if (o.clamp1) v = make_float2(fminf(v.x, 1.f), fminf(v.y, 1.f));
            }
            float* p = dz[z] + cols[c];
            if (PAIR) {
              *reinterpret_cast<float2*>(p + oA) = v;
            } else {
              p[oA] = v.x;
              p[oB] = v.y;
            }
          }
      }
      ox = ox + 1 == Ox ? 0 : ox + 1;
      col = after(ox, cols[1]);
      ox = ox + 1 == Ox ? 0 : ox + 1;
    }
#pragma unroll
    for (int fz = 0; fz < 2; ++fz)
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int p = 0; p < RW - 1; ++p) {
          wl[fz][y][p] = wl[fz][y][p + 1];
          wh[fz][y][p] = wh[fz][y][p + 1];
        }
  }
}

// Which compile-time bank a bank is: 1 bior1.5 x Haar, 2 Haar, 3 sym4 x Haar shape; 0 none.
static bool taps_are(const Taps& t, int first, int count) {
  if (t.n != count) return false;
  for (int u = 0; u < count; ++u)
    if (t.k[u] != first + u) return false;
  return true;
}

static int fast_kind(const WaveletBank& bk) {
  for (int f = 0; f < 2; ++f)
    if (!taps_are(bk.z.a[f], 0, 2) || !taps_are(bk.z.s[f], 0, 2)) return 0;
  auto is = [&](int al, int ah, int ahn, int sl, int sln, int sh) {
    return taps_are(bk.xy.a[0], 0, al) && taps_are(bk.xy.a[1], ah, ahn) && taps_are(bk.xy.s[0], sl, sln) &&
           taps_are(bk.xy.s[1], 0, sh);
  };
  return is(10, 4, 2, 4, 2, 10) ? 1 : is(2, 0, 2, 0, 2, 2) ? 2 : is(8, 0, 8, 0, 8, 8) ? 3 : 0;
}

static FastBank fast_bank(const WaveletBank& bk) {
  FastBank f{};
  auto put = [](float* d, const Taps& t) {
    for (int u = 0; u < t.n; ++u) d[u] = t.h[u];
  };
  put(f.alo, bk.xy.a[0]);
  put(f.ahi, bk.xy.a[1]);
  put(f.slo, bk.xy.s[0]);
  put(f.shi, bk.xy.s[1]);
  put(f.azl, bk.z.a[0]);
  put(f.azh, bk.z.a[1]);
  put(f.szl, bk.z.s[0]);
  put(f.szh, bk.z.s[1]);
  return f;
}

// Columns per march: long enough to amortise the halo steps (W / 2 columns in
// front), short enough to give every SM 32 warps: 4 instead of 8 columns at least took 128 x 96
// from 148 + 137 to 125 + 113 us; 64 warps per SM changed nothing.
static int march_segment(int len, long strips) {
  int seg = 64;
  while (seg > 4 && strips * ((len + seg - 1) / seg) < MARCH_WARPS) seg >>= 1;
  return seg;
}

template <int LL, int H0, int HN>
static cudaError_t launch_analysis_march(const float* in, int Ly, int Lx, int Lz, int shift, float* out,
                                         const FastBank& fb, const LevelBands& th, cudaStream_t st, int lo, int len,
                                         const SpinSet& sp) {
  const bool even = (shift & 1) == 0;
  const int nout = 32 - (imax(LL, H0 + HN) / 2 - (even ? 0 : 1));
  const int ty = (Ly / 2 + nout - 1) / nout, seg = march_segment(len, (long)ty * (Lz / 2) * sp.n);
  const dim3 grid((ty + MW - 1) / MW, (len + seg - 1) / seg, Lz / 2 * sp.n);
  auto kern = even ? k_wav_analysis_march<LL, H0, HN, true> : k_wav_analysis_march<LL, H0, HN, false>;
  launch_next(kern, grid, 32 * MW, 0, st, in, Ly, Lx, Lz, shift, out, fb, th, ty, lo, len, seg, sp);
  return cudaGetLastError();
}

template <int S0, int SN, int SH>
static cudaError_t launch_synthesis_march(const float* bands, const float* approx, int Oy, int Ox, int Oz,
                                          const SynthOut& o, const FastBank& fb, cudaStream_t st, int lo, int len,
                                          const SpinSet& sp) {
  const int ty = (Oy / 2 + 31) / 32, seg = march_segment(len, (long)ty * (Oz / 2) * sp.n);
  const dim3 grid((ty + MW - 1) / MW, (len + seg - 1) / seg, Oz / 2 * sp.n);
  const bool pair = (o.shift & 1) == 0;
  auto kern = o.first ? (pair ? k_wav_synthesis_march<S0, SN, SH, false, true> : k_wav_synthesis_march<S0, SN, SH, false, false>)
                      : (pair ? k_wav_synthesis_march<S0, SN, SH, true, true> : k_wav_synthesis_march<S0, SN, SH, true, false>);
  launch_next(kern, grid, 32 * MW, 0, st, bands, approx, Oy, Ox, Oz, o, fb, ty, lo, len, seg, sp);
  return cudaGetLastError();
}

// k_ht_weights for patches 16 and 32, one CTA per group: the group's slots are staged
// in shared memory ([k][c][r], 16-byte copies), then one warp adds each of the
// three terms, so the terms' serial chains run side by side.  Each is the
// same fixed-order reduction as in the generic kernel and the oracle: lane l adds
// the elements l, l + 32, ... of the column-major difference array (indices advanced by 32
// with carries), then an xor butterfly.  One warp per group, slot by slot, took
// 44 us for the 48 groups of 128 x 96 (here 8) and 82 us for a 720p frame's 920
// (here 51: 64 KB of slots allow three CTAs per SM, and each chain has 464 adds).
// GM: V is group-major (SynthOut), else image-shaped m x n x K (m a multiple of D).
template <int D, bool GM>
__global__ void __launch_bounds__(96) k_ht_weights_cta(const float* __restrict__ V, int m, int n, int M, int N, int K,
                                                       const int32_t* __restrict__ cnt, float* __restrict__ wgt,
                                                       int g0, int gn) {
  begin_after_previous(V, cnt);
  constexpr int DM = D - 3, SL = D * D;
  extern __shared__ __align__(16) float sg[];
  __shared__ float sum[3];
  const int term = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = window_group(blockIdx.x, g0, gn, M * N);
  if (g < 0) return;
  const int i = g % M, j = g / M;
  const int nm = cnt ? cnt[g] : K;
  const size_t ks = GM ? (size_t)SL : (size_t)m * n, cs = GM ? (size_t)D : (size_t)m;
  const float* base = GM ? V + (size_t)g * K * SL : V + (size_t)i * D + (size_t)j * D * m;
  for (int t = threadIdx.x; t < nm * (SL / 4); t += 96) {
    const int k = t / (SL / 4), c = t % (SL / 4) / (D / 4), r = 4 * (t % (D / 4));
    cp_async16(sg + 4 * t, base + ks * k + cs * c + r);
  }
  cp_async_wait_all();
  __syncthreads();
  float acc = 0.f;
  const int nx = D * DM * nm;
  if (term == 0) {  // x: element r + D (c + DM k)
    int c = lane / D;
    const float* q = sg + lane;  // element (r, c, k)
#pragma unroll 8
    for (int e = lane; e < nx; e += 32) {
      acc = acc + fabsf(d3(q[0], q[D], q[2 * D], q[3 * D]));
      q += 32;
      c += 32 / D;
      if (c >= DM) c -= DM, q += 3 * D;
    }
  } else if (term == 1) {  // y: element r + DM (c + D k)
    int r = lane % DM;
    const float* q = sg + (lane / DM) * D + r;
#pragma unroll 8
    for (int e = lane; e < nx; e += 32) {
      acc = acc + fabsf(d3(q[0], q[1], q[2], q[3]));
      q += (32 / DM) * D + 32 % DM;
      r += 32 % DM;
      if (r >= DM) r -= DM, q += D - DM;
    }
  } else {  // slots: element r + D (c + D k) of the pair (k, k + 1)
#pragma unroll 8
    for (int e = lane; e < (nm - 1) * SL; e += 32) acc = acc + fabsf(sg[e + SL] - sg[e]);
  }
  acc = warp_sum(acc);
  if (lane == 0) sum[term] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float w = sum[0] * 0.25f + sum[1] * 0.25f;
    w = w + sum[2];
    wgt[g] = 1.f / (w + 2.220446049250313e-16f);
  }
}

// medfilt3(Volume,[3 3 3]) (denoiseAndAggregateGPU.m:49-52) with 'symmetric'
// padding, which for a one-voxel border repeats the edge voxel.  The median
// of 27 values is a selection, exact in any order: an odd-even transposition
// sort in registers.
__global__ void __launch_bounds__(256) k_medfilt3(const float* __restrict__ V, int m, int n, int K,
                                                  float* __restrict__ out) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= (size_t)m * n * K) return;
  const int y = (int)(idx % m);
  const size_t r1 = idx / m;
  const int x = (int)(r1 % n), z = (int)(r1 / n);
  float v[27];
  int q = 0;
#pragma unroll
  for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
    for (int dx = -1; dx <= 1; ++dx)
#pragma unroll
      for (int dy = -1; dy <= 1; ++dy) {
        const int yy = min(max(y + dy, 0), m - 1), xx = min(max(x + dx, 0), n - 1), zz = min(max(z + dz, 0), K - 1);
        v[q++] = __ldg(V + yy + (size_t)m * (xx + (size_t)n * zz));
      }
#pragma unroll
  for (int pass = 0; pass < 27; ++pass)
#pragma unroll
    for (int i = pass & 1; i + 1 < 27; i += 2) {
      const float a = fminf(v[i], v[i + 1]), b = fmaxf(v[i], v[i + 1]);
      v[i] = a;
      v[i + 1] = b;
    }
  out[idx] = v[13];
}

cudaError_t launch_medfilt3(const float* V, int m, int n, int K, float* out, cudaStream_t st) {
  const size_t N = (size_t)m * n * K;
  k_medfilt3<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(V, m, n, K, out);
  return cudaGetLastError();
}

static size_t analysis_smem(int reach) {
  const int NY = 2 * TQ + reach;
  return (size_t)(2 * NY * NY + 4 * TQ * NY) * sizeof(float);
}

static size_t synthesis_smem(int reach) {
  const int NQ = (TP - 1 + reach) / 2 + 1;
  return (size_t)(8 * NQ * NQ + 4 * NQ * TP + 2 * TP * TP) * sizeof(float);
}

// The compile-time kernels take every size of at least the filter length (the
// generic ones drop taps past the end of a shorter axis).
static bool march_fits(int kind, int Ly, int Lx, int Lz) {
  const int W = kind == 1 ? 10 : kind == 2 ? 2 : 8;
  return kind && Ly >= W && Lx >= W && Lz >= 2 && Ly % 2 == 0 && Lx % 2 == 0 && Lz % 2 == 0;
}

cudaError_t launch_wav_analysis(const float* in, int Ly, int Lx, int Lz, int shift, float* out,
                                const WaveletBank& bk, const LevelBands& th, cudaStream_t st,
                                const ColRange& qcols, const SpinSet& sp) {
  const int kind = fast_kind(bk);
  if (march_fits(kind, Ly, Lx, Lz)) {
    const FastBank fb = fast_bank(bk);
    const int O = Lx / 2, lo = qcols.all(O) ? 0 : pmod(qcols.lo, O), len = qcols.all(O) ? O : qcols.len;
    if (len == 0) return cudaSuccess;
    if (kind == 1) return launch_analysis_march<10, 4, 2>(in, Ly, Lx, Lz, shift, out, fb, th, st, lo, len, sp);
    if (kind == 2) return launch_analysis_march<2, 0, 2>(in, Ly, Lx, Lz, shift, out, fb, th, st, lo, len, sp);
    return launch_analysis_march<8, 0, 8>(in, Ly, Lx, Lz, shift, out, fb, th, st, lo, len, sp);
  }
  const size_t sm = analysis_smem(bk.reach_a);
  cudaError_t e = cudaFuncSetAttribute(k_wav_analysis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  int t0, nt;
  tile_span(qcols, Lx / 2, TQ, t0, nt);
  if (nt == 0) return cudaSuccess;
  dim3 grid((Ly / 2 + TQ - 1) / TQ, nt, Lz / 2);
  for (int q = 0; q < sp.n; ++q)
    k_wav_analysis<<<grid, 256, sm, st>>>(in + q * sp.in, Ly, Lx, Lz, shift, out + q * sp.out, bk, th, t0);
  return cudaGetLastError();
}

cudaError_t launch_wav_synthesis(const float* bands, const float* approx, int Oy, int Ox, int Oz,
                                 const SynthOut& o, const WaveletBank& bk, cudaStream_t st,
                                 const ColRange& cols, const SpinSet& sp) {
  const int kind = fast_kind(bk);
  if (march_fits(kind, Oy, Ox, Oz)) {
    const FastBank fb = fast_bank(bk);
    // whole column pairs: the ones that hold the window's columns
    const int I = Ox / 2, first = pmod(cols.lo, Ox) / 2;
    const int pairs = cols.all(Ox) ? I : cols.len == 0 ? 0 : (pmod(cols.lo, Ox) + cols.len - 1) / 2 - first + 1;
    const int lo = pairs >= I ? 0 : first, len = pairs >= I ? I : pairs;
    if (len == 0) return cudaSuccess;
    if (kind == 1) return launch_synthesis_march<4, 2, 10>(bands, approx, Oy, Ox, Oz, o, fb, st, lo, len, sp);
    if (kind == 2) return launch_synthesis_march<0, 2, 2>(bands, approx, Oy, Ox, Oz, o, fb, st, lo, len, sp);
    return launch_synthesis_march<0, 8, 8>(bands, approx, Oy, Ox, Oz, o, fb, st, lo, len, sp);
  }
  const size_t sm = synthesis_smem(bk.reach_s);
  cudaError_t e = cudaFuncSetAttribute(k_wav_synthesis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  int t0, nt;
  tile_span(cols, Ox, TP, t0, nt);
  if (nt == 0) return cudaSuccess;
  dim3 grid((Oy + TP - 1) / TP, nt, Oz / 2);
  for (int q = 0; q < sp.n; ++q) {
    SynthOut oq = o;
    oq.out += q * sp.out;
    k_wav_synthesis<<<grid, 256, sm, st>>>(bands + q * sp.in, approx + q * sp.approx, Oy, Ox, Oz, oq, bk, t0);
  }
  return cudaGetLastError();
}

// k_ht_weights for patch 8: the whole group (nm slots of 8 x 8) is staged in
// shared memory slot-major ([k][c][r]), then each lane walks its elements
// e = lane + 32 t of the three difference arrays in increasing e, as the
// other versions do.  In that layout the slot term's element e sits at e and
// e + 64, and the x term's at e + 24 k (k = e / 40), so most of the per-term
// index arithmetic goes away.
template <bool GM>
__global__ void __launch_bounds__(128) k_ht_weights_8(const float* __restrict__ V, int m, int n, int M, int N,
                                                      int K, const int32_t* __restrict__ cnt,
                                                      float* __restrict__ wgt, int g0, int gn) {
  begin_after_previous(V, cnt);
  constexpr int D = 8, DM = D - 3, SL = D * D, SX = D * DM;
  extern __shared__ float shw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = window_group(blockIdx.x * 4 + warp, g0, gn, M * N);
  if (g < 0) return;
  float* sg = shw + warp * K * SL;
  const int i = g % M, j = g / M;
  const int nm = cnt ? cnt[g] : K;
  const size_t sz = GM ? (size_t)SL : (size_t)m * n;
  // lane: row r = lane % 8 of columns lane / 8 and lane / 8 + 4 of every slot
  const float* p0 = GM ? V + (size_t)g * K * SL + lane
                       : V + (size_t)i * D + (size_t)(j * D + (lane >> 3)) * m + (lane & 7);
  const float* p1 = p0 + (GM ? (size_t)32 : (size_t)4 * m);
  // slots in batches of 4: eight independent loads in flight per lane.  The slot
  // term's elements lane and lane + 32 of a pair (k - 1, k) are the lane's own values.
  float tx = 0.f, ty = 0.f, tz = 0.f;
  float pa = 0.f, pb = 0.f;
  auto slot = [&](int k, float a, float b) {
    sg[k * SL + lane] = a;
    sg[k * SL + 32 + lane] = b;
    if (k > 0) {
      tz = tz + fabsf(a - pa);
      tz = tz + fabsf(b - pb);
    }
    pa = a;
    pb = b;
  };
  int k = 0;
  for (; k + 4 <= nm; k += 4) {
    float a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      a[u] = __ldg(p0 + sz * (k + u));
      b[u] = __ldg(p1 + sz * (k + u));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) slot(k + u, a[u], b[u]);
  }
  for (; k < nm; ++k) slot(k, __ldg(p0 + sz * k), __ldg(p1 + sz * k));
  __syncwarp();
  // x term: element r + D (c + DM k) -> V(r, c .. c+3, k) at r + D c + SL k = e + (SL - SX) k
  for (int e = lane; e < nm * SX; e += 32) {
    const int k = e / SX;
    const float* q = sg + e + (SL - SX) * k;
    tx = tx + fabsf(d3(q[0], q[D], q[2 * D], q[3 * D]));
  }
  // y term: element r + DM (c + D k) -> V(r .. r+3, c, k)
  for (int e = lane; e < nm * SX; e += 32) {
    const int k = e / SX, rem = e - k * SX, c = rem / DM, r = rem - c * DM;
    const float* q = sg + k * SL + c * D + r;
    ty = ty + fabsf(d3(q[0], q[1], q[2], q[3]));
  }
  tx = warp_sum(tx);
  ty = warp_sum(ty);
  tz = warp_sum(tz);
  if (lane == 0) {
    float w = tx * 0.25f + ty * 0.25f;
    w = w + tz;
    wgt[g] = 1.f / (w + 2.220446049250313e-16f);
  }
}

cudaError_t launch_ht_weights(const float* Vavg, int m, int n, int M, int N, int d, int K,
                              const int32_t* cnt, float* wgt, cudaStream_t st, const ColRange& jcols,
                              bool group_major) {
  int g0, gn;
  group_span(jcols, M, N, g0, gn);
  if (gn < 0) return cudaSuccess;
  const int G = gn > 0 ? gn : M * N;
  if (d == 8) {
    const size_t smb = (size_t)4 * K * 64 * sizeof(float);
    auto kern = group_major ? k_ht_weights_8<true> : k_ht_weights_8<false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb);
    if (e != cudaSuccess) return e;
    launch_next(kern, (G + 3) / 4, 128, smb, st, Vavg, m, n, M, N, K, cnt, wgt, g0, gn);
  } else if (d == 16 || (d == 32 && !group_major)) {
    auto kern = d == 32 ? k_ht_weights_cta<32, false> : group_major ? k_ht_weights_cta<16, true> : k_ht_weights_cta<16, false>;
    const size_t smb = (size_t)K * d * d * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smb);
    if (e != cudaSuccess) return e;
    launch_next(kern, G, 96, smb, st, Vavg, m, n, M, N, K, cnt, wgt, g0, gn);
  } else if (group_major) {
    return cudaErrorInvalidValue;
  } else {
    k_ht_weights<<<(G + 3) / 4, 128, 0, st>>>(Vavg, m, n, M, N, d, K, cnt, wgt, g0, gn);
  }
  return cudaGetLastError();
}

}  // namespace gbm3d

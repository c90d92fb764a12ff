// Deterministic owner-computes aggregation — denoiseAndAggregateGPU.m:58-92 (loop :70-89)
// and denoiseAndAggregateWieFast.m:84-100.
//
// The reference adds every matched block, weighted, into U and W in the loop
// order (reference row y, reference column x, match i), each add rounded to
// single.  Here each output pixel is owned by one lane, which applies its
// contributions in exactly that order, so the result is bit-identical to the
// sequential loop and needs no atomics.
//
// Contributions falling outside the cropped image are never produced (the
// reference crops them away, denoiseAndAggregateGPU.m:91-92).
#include "common.cuh"
#include "kernels.cuh"

namespace gbm3d {

__host__ __device__ inline int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }
__host__ __device__ inline int ceil_div(int a, int b) { return -floor_div(-a, b); }

constexpr int TR = 8, TC = 4;  // warp tile: 8 rows (fast axis) x 4 columns, one pixel per lane
constexpr int LCAP = 96;       // list chunk per warp (entries); walked whenever it may overflow
constexpr int BIAS = 1 << 12;  // offset added to tile-relative block origins before packing

// A CTA of 8 warps owns CR x CC output pixels (16 warp tiles of TR x TC, two
// per warp, one pixel per lane).
//  1. The CTA enumerates the candidates (reference i, j, slot k) whose search
//     window reaches its pixels, in the reference's loop order, 256 per
//     round, and compacts the blocks that intersect its pixels into a
//     shared-memory list in that order (warp ballots, then the warps' counts
//     in warp order).
//  2. Each warp filters the CTA list, in order, for the entries touching one
//     of its warp tiles, computing for each the mask of lanes it covers and
//     the lane-independent part of its offsets (a warp list of at most LCAP
//     entries, walked whenever it may overflow).
//  3. The walk: all lanes step through the warp list together, WB entries at
//     a time; a covered lane loads its element and adds the contribution.
// Every pixel receives its contributions in the reference's order, so the
// sums are bit-identical to the sequential loop.
//   step 1: value (wg * Vavg) * mask, weight wg * mask   (denoiseAndAggregateGPU.m:84-85)
//   step 2: value and weight precomputed by the Wiener kernel (:84-90 of
//           denoiseAndAggregateWieFast.m), the same single-precision products
constexpr int CR = 32, CC = 16;                    // CTA pixel tile
constexpr int NSR = CR / TR, NSC = CC / TC;        // warp tiles per CTA tile: 4 x 4
constexpr int NTC = 256;                           // threads per CTA
constexpr int SUBS = NSR * NSC / (NTC / 32);       // warp tiles per warp: 2
constexpr int WB = 8;                              // walk batch: entries tested and loaded together

// CAPC: CTA list capacity (entries).  A list that would overflow is walked in
// order and refilled, so any capacity gives the same sums; a small one suits
// sparse reference grids (fewer entries per tile) and lets more CTAs reside.
template <int D, int D2, bool WIE, bool KAHAN, int CAPC>
__global__ void __launch_bounds__(NTC) k_aggregate_cta(AggArgs A) {
  const float* blocks = A.blocks;
  const float* gw = A.gw;
  const uint32_t* Sg = A.S;
  const int32_t* counts = A.cnt;
  begin_after_previous(blocks, gw, Sg, counts);
  extern __shared__ int smi[];
  __shared__ int wcnt[NTC / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  float* win = reinterpret_cast<float*>(smi);
  int4* lstC = reinterpret_cast<int4*>(smi + ((D * D + 3) & ~3));
  int4* lst = lstC + CAPC + warp * LCAP;
  if (!WIE)
    for (int t = tid; t < D * D; t += NTC) win[t] = A.win[t];
  const int tiles_r = (A.m + CR - 1) / CR, tiles_c = (A.n + CC - 1) / CC;
  const int tcol = (int)(blockIdx.x / tiles_r) + A.ct0;  // the window's column tiles, modulo the count
  const int R0 = (blockIdx.x % tiles_r) * CR, C0 = (tcol >= tiles_c ? tcol - tiles_c : tcol) * CC;
  const int K = A.K, s = A.s;
  const int mv = A.M * D;
  constexpr int H = D2 / 2;
  const int PR0 = R0 + H, PC0 = C0 + H;
  const int i_lo = max(0, ceil_div(PR0 - D - D2 + 2, s)), i_hi = min(A.M - 1, floor_div(PR0 + CR - 1, s));
  const int j_lo = max(0, ceil_div(PC0 - D - D2 + 2, s)), j_hi = min(A.N - 1, floor_div(PC0 + CC - 1, s));
  const int NI = i_hi - i_lo + 1, NJ = j_hi - j_lo + 1;
  const int total = (NI > 0 && NJ > 0) ? NI * NJ * K : 0;
  const unsigned invK = K > 1 ? (unsigned)(0xFFFFFFFFu / (unsigned)K) + 1u : 0u;  // ceil(2^32 / K)
  const unsigned invNJ = NJ > 1 ? (unsigned)(0xFFFFFFFFu / (unsigned)NJ) + 1u : 0u;
  const size_t mn = (size_t)mv * (A.N * D);
  const unsigned FULL = 0xffffffffu;

  // this lane's pixel in each of the warp's tiles (CTA-relative)
  const int pr = lane & 7, pc = lane >> 3;
  int prc[SUBS], pcc[SUBS];
  float u[SUBS], w[SUBS], cu[SUBS], cw[SUBS];
#pragma unroll
  for (int a = 0; a < SUBS; ++a) {
    const int sid = warp + (NTC / 32) * a;
    prc[a] = (sid % NSR) * TR + pr;
    pcc[a] = (sid / NSR) * TC + pc;
    u[a] = w[a] = cu[a] = cw[a] = 0.f;
  }
  auto add = [&](float& acc, float& comp, float x) {
    if (KAHAN) {
      const float y = x - comp;
      const float t = acc + y;
      comp = (t - acc) - y;
      acc = t;
    } else {
      acc = acc + x;
    }
  };
  // Warp-list entries carry what the lanes need precomputed for their warp
  // tile: x = the 32-bit mask of lanes whose pixel the block covers, y and z
  // the offsets of the block's data and weights minus the lane-independent
  // part, w the group weight (step 1).  A lane's element is then y + a lane
  // constant.  All lanes step through the entries together (the loads of one
  // entry fall in a few sectors); uncovered lanes skip the adds.
  const int voff = WIE ? pr + pc * D : pr + mv * pc;  // lane offset in a block's data
  const int woff = pr + pc * D;                       // lane offset in a d x d table
  auto walk = [&](int a, int count) {
    for (int e0 = 0; e0 < count; e0 += WB) {  // the list is padded to WB with empty masks
      int4 en[WB];
      bool cov[WB];
      float val[WB], wv[WB];
#pragma unroll
      for (int t = 0; t < WB; ++t) {
        en[t] = lst[e0 + t];
        cov[t] = (en[t].x >> lane) & 1;
        val[t] = cov[t] ? __ldg(blocks + ((size_t)(unsigned)(en[t].y + voff))) : 0.f;
        if (WIE) wv[t] = cov[t] ? __ldg(gw + ((size_t)(unsigned)(en[t].z + woff))) : 0.f;
        else wv[t] = cov[t] ? win[woff - en[t].z] : 0.f;
      }
#pragma unroll
      for (int t = 0; t < WB; ++t) {
        if (cov[t]) {
          if (WIE) {
            add(u[a], cu[a], val[t]);
            add(w[a], cw[a], wv[t]);
          } else {
            const float wg = __int_as_float(en[t].w);
            add(u[a], cu[a], (wg * val[t]) * wv[t]);
            add(w[a], cw[a], wg * wv[t]);
          }
        }
      }
    }
  };
  // every warp: its tiles' entries of the CTA list, in order, converted to
  // warp-list entries (mask and warp-tile-relative offsets)
  auto process = [&](int count) {
#pragma unroll
    for (int a = 0; a < SUBS; ++a) {
      const int sr = prc[a] - pr, sc = pcc[a] - pc;  // warp tile origin (CTA-relative)
      int cnt = 0;
      auto flush = [&]() {
        const int pad = (WB - (cnt % WB)) % WB;  // empty entries up to a multiple of WB
        if (lane < pad) lst[cnt + lane] = make_int4(0, 0, 0, 0);
        __syncwarp();
        walk(a, cnt + pad);
        __syncwarp();
        cnt = 0;
      };
      for (int e0 = 0; e0 < count; e0 += 32) {
        const int e = e0 + lane;
        bool hit = false;
        int4 en = make_int4(0, 0, 0, 0);
        if (e < count) {
          const int4 ec = lstC[e];
          const int r0 = (ec.x & 0xffff) - BIAS - sr, c0 = (ec.x >> 16) - BIAS - sc;  // warp-tile-relative origin
          const int rlo = max(r0, 0), rhi = min(r0 + D, TR), clo = max(c0, 0), chi = min(c0 + D, TC);
          hit = rhi > rlo && chi > clo;
          if (hit) {
            const unsigned rows = ((1u << rhi) - 1u) & ~((1u << rlo) - 1u);
            const unsigned cols = ((1u << chi) - 1u) & ~((1u << clo) - 1u);
            const unsigned spread = (cols & 1u) | ((cols & 2u) << 7) | ((cols & 4u) << 14) | ((cols & 8u) << 21);
            en.x = (int)(rows * spread);  // lane pr + 8 pc covered iff row pr and column pc are
            if (WIE) {
              en.y = ec.y - r0 - c0 * D;
              en.z = ec.z - r0 - c0 * D;
            } else {
              en.y = ec.y - r0 - mv * c0;
              en.z = r0 + c0 * D;
              en.w = ec.z;
            }
          }
        }
        const unsigned bal = __ballot_sync(FULL, hit);
        if (hit) lst[cnt + __popc(bal & ((1u << lane) - 1u))] = en;
        cnt += __popc(bal);
        if (cnt > LCAP - 32 - WB) flush();
      }
      flush();
    }
  };

  __syncthreads();  // win
  int countC = 0;
  for (int base = 0; base < total; base += NTC) {
    const int q = base + tid;
    bool hit = false;
    int4 ent = make_int4(0, 0, 0, 0);
    if (q < total) {
      // q / K and r2 / NJ by multiply-high with ceil(2^32 / divisor): exact
      // for dividends below 2^32 / divisor (here below NI NJ K < 2^20)
      const int r2 = K > 1 ? (int)__umulhi((unsigned)q, invK) : q, k = q - r2 * K;
      const int i2 = NJ > 1 ? (int)__umulhi((unsigned)r2, invNJ) : r2;
      const int i = i_lo + i2, j = j_lo + (r2 - i2 * NJ);
      const int g = i + A.M * j;
      // the count, the match index and the group weight are independent
      // loads: all three in flight before the count test (S holds K entries
      // per group whatever the count)
      const int nm = counts ? __ldg(counts + g) : K;
      const int eS = (int)__ldg(Sg + (size_t)g * K + k) - 1;
      const float gwv = WIE ? 0.f : __ldg(gw + g);
      if (k < nm) {
        const int e = eS;
        const int r0 = i * s + e % D2 - PR0, c0 = j * s + e / D2 - PC0;
        hit = r0 < CR && r0 + D > 0 && c0 < CC && c0 + D > 0;
        if (hit) {
          ent.x = (r0 + BIAS) | ((c0 + BIAS) << 16);
          if (WIE) {
            ent.y = (g * K + k) * (D * D);
            ent.z = g * (D * D);
          } else {
            ent.y = (int)((size_t)i * D + (size_t)mv * (j * D) + mn * k);
            ent.z = __float_as_int(gwv);
          }
        }
      }
    }
    const unsigned bal = __ballot_sync(FULL, hit);
    if (lane == 0) wcnt[warp] = __popc(bal);
    __syncthreads();
    int off = countC, tot = 0;
#pragma unroll
    for (int v = 0; v < NTC / 32; ++v) {
      off += v < warp ? wcnt[v] : 0;
      tot += wcnt[v];
    }
    if (hit) lstC[off + __popc(bal & ((1u << lane) - 1u))] = ent;
    countC += tot;
    __syncthreads();
    if (countC > CAPC - NTC) {
      process(countC);
      countC = 0;
      __syncthreads();
    }
  }
  process(countC);
#pragma unroll
  for (int a = 0; a < SUBS; ++a) {
    const int orow = R0 + prc[a], ocol = C0 + pcc[a];
    if (orow < A.m && ocol < A.n) {
      A.U[orow + (size_t)A.m * ocol] = u[a];
      A.W[orow + (size_t)A.m * ocol] = w[a];
    }
  }
}

template <int D, int D2, bool WIE, bool KAHAN, int CAPC>
static cudaError_t launch_px_cap(const AggArgs& A, cudaStream_t st) {
  const size_t sm = (size_t)((D * D + 3) & ~3) * sizeof(float) + (size_t)(CAPC + (NTC / 32) * LCAP) * sizeof(int4);
  cudaError_t e = cudaFuncSetAttribute(k_aggregate_cta<D, D2, WIE, KAHAN, CAPC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  AggArgs B = A;
  int nt;
  tile_span(A.cols, A.n, CC, B.ct0, nt);
  if (nt == 0) return cudaSuccess;
  const int tiles = ((A.m + CR - 1) / CR) * nt;
  launch_next(k_aggregate_cta<D, D2, WIE, KAHAN, CAPC>, tiles, NTC, sm, st, B);
  return cudaGetLastError();
}

// The same owner-ordered sums, a block at a time (patches 8 and 16).  The
// kernel above steps the lanes of an 8 x 4 pixel tile through every block that
// touches the tile: 39 % of its lane slots add something, and every warp filters
// its CTA's list once per tile.  Here one warp owns RR x RC pixels whose (U, W)
// sums sit in shared memory, and each lane stands for fixed pixels of the
// *block*: an entry is one load of the block, and a read, two adds per pixel
// and a write of the sums, with every lane at work.  The warp applies its entries one
// after another in the reference's loop order, so every pixel receives the
// same contributions in the same order and the sums are unchanged.
//   The region has a border of D pixels in front and D - 1 behind, so a block
// that overlaps it needs no test per pixel; sums of border pixels are never
// written out (their owners make them).
//   PT, the region's column pitch, is 8 modulo 16 pixels of eight bytes: the
// 8 x 4 pixels of a half patch fall on distinct banks at every block offset.
//   The warp enumerates the candidates (reference i, j, slot k) whose search
// window reaches its region, in loop order.  A block is
// 256 (1024) contiguous bytes (group-major), two lines where the image-shaped
// volume has eight, and is prefetched into L2 when it is listed.
//   A region of 8 x 8 runs where the GPU is not full (301 x 203: 1.7 warps per
// scheduler, each issuing one instruction in seven cycles), so there a second warp makes
// list r + 1 while the first walks list r: 322 -> 278 us for the four launches of
// 301 x 203.  On the larger regions the second warp takes slots from other regions
// (16 x 16: 512^2 126 -> 168 us; 24 x 24: 4096^2 1.15 -> 1.81 ms).
//   Bounds at 1024^2 dense (ncu): shared-memory pipe 61 %, issue 42-50 %, DRAM
// 33 %; 272 us per launch against 625 us pixel at a time (of which the
// group-major layout with its prefetch 310: DRAM reads 2.07 -> 0.72 GB).

// N floats at p (a multiple of 128 bytes) on their way to L2: an entry's block
// is loaded only when the list is walked.
template <int N>
__device__ __forceinline__ void prefetch_l2(const float* p) {
#pragma unroll
  for (int t = 0; t < N; t += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + t));
}

template <int D, bool KAHAN, int RR, int RC>
struct AggBlk {
  static constexpr int PT = D == 8 ? ((RR + 2 * D - 1 + 7) / 16) * 16 + 8 : RR + 2 * D - 1;
  static constexpr int COLS = RC + 2 * D - 1;
  static constexpr int SV = KAHAN ? 4 : 2;  // floats per pixel: u, w (and their compensations)
  static constexpr int NB = D == 8 ? 8 : 4; // entries loaded together
  static constexpr int EB = 4;              // candidates per lane and enumeration round
  static constexpr bool TWO = RR <= 8;      // one warp lists, the other walks
  static constexpr int NT = TWO ? 64 : 32;
  static constexpr int LC = (TWO ? 96 : 128) + 32 * EB;  // list capacity
  static constexpr int LISTS = (TWO ? 2 : 1) * (LC + 2 * NB);
  static constexpr int CELLS4 = (PT * COLS * SV + 3) / 4;  // the sums in 16-byte words
  static constexpr size_t BYTES = (size_t)LISTS * sizeof(int4) + (size_t)CELLS4 * sizeof(float4);
  static_assert(PT >= RR + 2 * D - 1, "pitch");
};

template <int D, int D2, bool WIE, bool KAHAN, int RR, int RC>
__global__ void __launch_bounds__(AggBlk<D, KAHAN, RR, RC>::NT) k_aggregate_blk(AggArgs A) {
  const float* blocks = A.blocks;
  const float* gw = A.gw;
  const uint32_t* Sg = A.S;
  const int32_t* counts = A.cnt;
  begin_after_previous(blocks, gw, Sg, counts);
  using G = AggBlk<D, KAHAN, RR, RC>;
  constexpr int PT = G::PT, SV = G::SV, NB = G::NB, EB = G::EB;
  constexpr int NP = D * D / 32, CSTEP = 32 / D;  // pixels per lane, block columns between them
  constexpr int H = D2 / 2;
  extern __shared__ int4 smv[];
  const int lane = threadIdx.x & 31;
  const bool walks = !G::TWO || threadIdx.x < 32, lists = !G::TWO || threadIdx.x >= 32;
  int4* lst = smv;
  float* acc = reinterpret_cast<float*>(smv + G::LISTS);
  const unsigned FULL = 0xffffffffu, below = (1u << lane) - 1u;
  for (int e = threadIdx.x; e < G::CELLS4; e += G::NT) reinterpret_cast<float4*>(acc)[e] = make_float4(0.f, 0.f, 0.f, 0.f);

  const int tiles_r = (A.m + RR - 1) / RR, tiles_c = (A.n + RC - 1) / RC;
  const int tcol = (int)(blockIdx.x / tiles_r) + A.ct0;  // the window's column tiles, modulo the count
  const int R0 = (blockIdx.x % tiles_r) * RR, C0 = (tcol >= tiles_c ? tcol - tiles_c : tcol) * RC;
  const int K = A.K, s = A.s;
  const int PR0 = R0 + H, PC0 = C0 + H;
  const int i_lo = max(0, ceil_div(PR0 - D - D2 + 2, s)), i_hi = min(A.M - 1, floor_div(PR0 + RR - 1, s));
  const int j_lo = max(0, ceil_div(PC0 - D - D2 + 2, s)), j_hi = min(A.N - 1, floor_div(PC0 + RC - 1, s));
  const int NI = i_hi - i_lo + 1, NJ = j_hi - j_lo + 1;
  const int total = (NI > 0 && NJ > 0) ? NI * NJ * K : 0;
  const unsigned invK = K > 1 ? (unsigned)(0xFFFFFFFFu / (unsigned)K) + 1u : 0u;  // ceil(2^32 / K)
  const unsigned invNJ = NJ > 1 ? (unsigned)(0xFFFFFFFFu / (unsigned)NJ) + 1u : 0u;

  // this lane's block pixels: (pr, pc + CSTEP q)
  const int pr = lane % D, pc = lane / D;
  const float* vsrc = blocks + lane;
  const float* wsrc = WIE ? gw + lane : nullptr;
  float* apx = acc + (pr + PT * pc) * SV;
  float mask[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) mask[q] = WIE ? 0.f : A.win[lane + 32 * q];

  struct Batch {
    int off[NB];  // the block's place in acc
    float wg[NB], val[NB][NP], wv[NB][WIE ? NP : 1];
  };
  auto fetch = [&](Batch& B, int e0) {
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      const int4 en = lst[e0 + t];
      B.off[t] = en.x;
      if (!WIE) B.wg[t] = __int_as_float(en.z);
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        B.val[t][q] = __ldg(vsrc + (size_t)(unsigned)(en.y + 32 * q));
        if (WIE) B.wv[t][q] = __ldg(wsrc + (size_t)(unsigned)(en.z + 32 * q));
      }
    }
  };
  auto add = [](float& a, float& comp, float x) {
    const float y = x - comp;
    const float t = a + y;
    comp = (t - a) - y;
    a = t;
  };
  auto apply = [&](const Batch& B) {
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      float* p = apx + B.off[t];
      float dv[NP], dw[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        dv[q] = WIE ? B.val[t][q] : (B.wg[t] * B.val[t][q]) * mask[q];
        dw[q] = WIE ? B.wv[t][WIE ? q : 0] : B.wg[t] * mask[q];
      }
      if constexpr (KAHAN) {
        float4 v[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) v[q] = *reinterpret_cast<float4*>(p + PT * CSTEP * q * SV);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          add(v[q].x, v[q].z, dv[q]);
          add(v[q].y, v[q].w, dw[q]);
          *reinterpret_cast<float4*>(p + PT * CSTEP * q * SV) = v[q];
        }
      } else {
        float2 v[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) v[q] = *reinterpret_cast<float2*>(p + PT * CSTEP * q * SV);
#pragma unroll
        for (int q = 0; q < NP; ++q)
          *reinterpret_cast<float2*>(p + PT * CSTEP * q * SV) = make_float2(v[q].x + dv[q], v[q].y + dw[q]);
      }
      __syncwarp();  // the next entry's pixels may be other lanes' of this one
    }
  };
  // the list, in order; padded to whole batches with entries on the border (offset 0: rows and columns -D .. -1)
  auto walk = [&](int count) {
    if (lane < 2 * NB) lst[count + lane] = make_int4(0, 0, 0, 0);
    __syncwarp();
    Batch B0, B1;
    fetch(B0, 0);
    for (int e0 = 0; e0 < count; e0 += 2 * NB) {
      fetch(B1, e0 + NB);
      apply(B0);
      if (e0 + 2 * NB < count) fetch(B0, e0 + 2 * NB);
      apply(B1);
    }
    __syncwarp();
  };

  // a round's candidates: index q of the loop order -> (i, j, k), its match
  // index, its group's count and weight; the next round's loads are in flight
  // while a round is tested
  struct Cand {
    int e[EB], nm[EB];
    float gw[EB];
  };
  auto decode = [&](int q, int& i, int& j, int& k) {
    // q / K and r2 / NJ by multiply-high with ceil(2^32 / divisor): exact for
    // dividends below 2^32 / divisor (here below NI NJ K < 2^20)
    const int r2 = K > 1 ? (int)__umulhi((unsigned)q, invK) : q;
    const int i2 = NJ > 1 ? (int)__umulhi((unsigned)r2, invNJ) : r2;
    k = q - r2 * K;
    i = i_lo + i2;
    j = j_lo + (r2 - i2 * NJ);
  };
  auto look = [&](Cand& C, int base) {
#pragma unroll
    for (int u = 0; u < EB; ++u) {
      int i, j, k;
      decode(min(base + 32 * u + lane, total - 1), i, j, k);
      const int g = i + A.M * j;
      C.nm[u] = counts ? __ldg(counts + g) : K;
      C.e[u] = (int)__ldg(Sg + (size_t)g * K + k) - 1;
      C.gw[u] = WIE ? 0.f : __ldg(gw + g);
    }
  };
  // the entries of candidates base, base + 1, ... until the list may be full
  int base = 0;
  Cand next;
  if (lists && total > 0) look(next, 0);
  auto fill = [&]() {
    int cnt = 0;
    for (; base < total && cnt <= G::LC - 32 * EB; base += 32 * EB) {
      const Cand cur = next;
      if (base + 32 * EB < total) look(next, base + 32 * EB);
#pragma unroll
      for (int u = 0; u < EB; ++u) {
        int i, j, k;
        decode(min(base + 32 * u + lane, total - 1), i, j, k);
        const int e = cur.e[u], r0 = i * s + e % D2 - PR0, c0 = j * s + e / D2 - PC0;
        const bool hit = base + 32 * u + lane < total && k < cur.nm[u] && r0 > -D && r0 < RR && c0 > -D && c0 < RC;
        const unsigned bal = __ballot_sync(FULL, hit);
        if (hit) {
          const int g = i + A.M * j;
          int4 en;
          en.x = (r0 + D + PT * (c0 + D)) * SV;
          en.y = (g * K + k) * (D * D);
          en.z = WIE ? g * (D * D) : __float_as_int(cur.gw[u]);
          en.w = 0;
          lst[cnt + __popc(bal & below)] = en;
          prefetch_l2<D * D>(blocks + (size_t)(unsigned)en.y);
        }
        cnt += __popc(bal);
      }
    }
    return cnt;
  };
  if constexpr (G::TWO) {
    // list r + 1 is made while list r is walked; one barrier per list
    __shared__ int scnt[2];
    for (int r = 0;; ++r) {
      lst = smv + (r & 1) * (G::LC + 2 * NB);
      if (lists) {
        const int cnt = fill();
        if (lane == 0) scnt[r & 1] = base < total ? cnt : -1 - cnt;  // negative: the last one
      }
      __syncthreads();
      const int c = scnt[r & 1], cnt = c < 0 ? -1 - c : c;
      if (walks && cnt) walk(cnt);
      if (c < 0) break;
    }
    __syncthreads();
  } else {
    __syncwarp();
    while (base < total) {
      const int cnt = fill();
      if (cnt) walk(cnt);
    }
    __syncwarp();
  }
  for (int e = threadIdx.x; e < RR * RC; e += G::NT) {
    const int r = e % RR, c = e / RR, orow = R0 + r, ocol = C0 + c;
    if (orow < A.m && ocol < A.n) {
      const float2 v = *reinterpret_cast<const float2*>(acc + (r + D + PT * (c + D)) * SV);
      A.U[orow + (size_t)A.m * ocol] = v.x;
      A.W[orow + (size_t)A.m * ocol] = v.y;
    }
  }
}

template <int D, int D2, bool WIE, bool KAHAN, int RR, int RC>
static cudaError_t launch_blk(const AggArgs& A, cudaStream_t st) {
  constexpr size_t sm = AggBlk<D, KAHAN, RR, RC>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(k_aggregate_blk<D, D2, WIE, KAHAN, RR, RC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  AggArgs B = A;
  int nt;
  tile_span(A.cols, A.n, RC, B.ct0, nt);
  if (nt == 0) return cudaSuccess;
  launch_next(k_aggregate_blk<D, D2, WIE, KAHAN, RR, RC>, ((A.m + RR - 1) / RR) * nt,
              AggBlk<D, KAHAN, RR, RC>::NT, sm, st, B);
  return cudaGetLastError();
}

// Patches 8 and 16 with group-major blocks: block at a time, on the largest
// region that still gives every SM enough warps to cover the latency of its
// entries' chain: 24 x 24 (13 resident warps per SM by shared memory) from 10
// regions per SM on, 16 x 16 from 5, else 8 x 8.  Smaller regions touch more
// entries per pixel (at stride 8: 0.42 per pixel at 24, 0.52 at 16, 0.88 at 8) but
// fill the GPU.  Measured, all aggregations of a call in us (pixel-at-a-time
// kernel / 24 / 16 / 8 with one warp): 4096^2 at strides 8 / 7 2232 / 1177 / 1394 / 2791; 1024^2
// dense 2502 / 1190 / 1340 / 2042; 512^2 reference tiling 131 / 146 / 125 / 175; 301 x 203
// dense 590 / 730 / 465 / 318 (two warps 278); 128 x 96 77 / 106 / 82 / 69 (67).
// Otherwise (the median filter's image-shaped volume, other patches): pixel at
// a time, with the list capacity from the expected entries of a tile:
// (candidate references across the tile's reach) x K, about a quarter of which
// touch the tile.
template <int D, int D2, bool WIE, bool KAHAN = false>
static cudaError_t launch_px(const AggArgs& A, cudaStream_t st) {
  if constexpr (D == 8 || D == 16) {
    if (A.group_major) {
      auto regions = [&](int r) { return (long)((A.m + r - 1) / r) * ((A.n + r - 1) / r); };
      if (regions(24) >= 10 * 148) return launch_blk<D, D2, WIE, KAHAN, 24, 24>(A, st);
      if (regions(16) >= 5 * 148) return launch_blk<D, D2, WIE, KAHAN, 16, 16>(A, st);
      return launch_blk<D, D2, WIE, KAHAN, 8, 8>(A, st);
    }
  }
  if constexpr (WIE && (D == 8 || D == 16)) {
    return cudaErrorInvalidValue;  // step 2's blocks are always group-major
  } else {
    if (!WIE && A.group_major) return cudaErrorInvalidValue;
    const long refs = (long)((CR + D + D2 - 2) / A.s + 1) * ((CC + D + D2 - 2) / A.s + 1);
    if (refs * A.K / 4 <= 1024 - NTC) return launch_px_cap<D, D2, WIE, KAHAN, 1024>(A, st);
    return launch_px_cap<D, D2, WIE, KAHAN, 2048>(A, st);
  }
}

cudaError_t launch_aggregate(const AggArgs& A, cudaStream_t st) {
  // block data offsets are 32-bit in the list entries
  if ((size_t)A.m * A.n * A.K >= ((size_t)1 << 31) || (size_t)A.M * A.N * A.K * A.d * A.d >= ((size_t)1 << 31) ||
      A.s < 1 || A.s > A.d)
    return cudaErrorInvalidValue;
  if (A.kahan) {  // precision form: patch 8
#define GBM3D_AGGK_CASE(DD2) \
  if (A.d == 8 && A.d2 == DD2) return A.wiener ? launch_px<8, DD2, true, true>(A, st) : launch_px<8, DD2, false, true>(A, st);
    GBM3D_AGGK_CASE(16) GBM3D_AGGK_CASE(24) GBM3D_AGGK_CASE(32)
#undef GBM3D_AGGK_CASE
    return cudaErrorInvalidValue;
  }
#define GBM3D_AGG_CASE(DD, DD2)                                                                 \
  if (A.d == DD && A.d2 == DD2)                                                                 \
    return A.wiener ? launch_px<DD, DD2, true>(A, st) : launch_px<DD, DD2, false>(A, st);
  GBM3D_AGG_CASE(8, 16) GBM3D_AGG_CASE(8, 24) GBM3D_AGG_CASE(8, 32)
  GBM3D_AGG_CASE(16, 16) GBM3D_AGG_CASE(16, 24) GBM3D_AGG_CASE(16, 32)
  GBM3D_AGG_CASE(32, 16) GBM3D_AGG_CASE(32, 24) GBM3D_AGG_CASE(32, 32)
  GBM3D_AGG_CASE(4, 16) GBM3D_AGG_CASE(4, 24) GBM3D_AGG_CASE(4, 32)
#undef GBM3D_AGG_CASE
  return cudaErrorInvalidValue;
}

}  // namespace gbm3d

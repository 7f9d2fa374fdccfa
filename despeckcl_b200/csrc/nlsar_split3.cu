// NL-SAR on 3x3 covariances with every similarity and weight computed once:
// the results of nlsar3_fast_kernel (nlsar_dim3.cu), bit for bit, from
//
//  sim3_kernel    per scale, the similarities of the lower half window into a
//      volume in memory.  A 3x3 similarity reads twenty words and costs about
//      three times a 2x2 one; computed here it is evaluated once per pixel
//      pair with no patch halo (the fused kernel: twice, with a 2.1x halo on
//      its 32 x 8 tiles), and the centre stays in registers over all offsets.
//  words3_kernel  from those, the patch sums and weight codes of a pass
//      (WordWalk, as in nlsar_split.cu).
//  mean3_kernel   per output pixel, all offsets in the reference's row-major
//      order: the weights of both halves, 23 accumulators per patch size, then
//      selection and blended output.
//
// The fused kernel spent 4.57 ms on 509 x 512 with patches {3,5,7} and scales
// {1,3}.
//
// Settings of the general kernel (nlsar3_kernel: other windows, patches {3,5},
// 9 or 11 alone) take the same three steps with its arithmetic and summation
// order, for its bits (EXACT, exact3_mean_kernel): 280 x 290 with {3,5,7} and
// search 15 3.72 -> 0.82 ms, search 23 8.60 -> 1.72 ms, {3,5} and search 21
// 5.30 -> 1.23 ms.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "dcl_internal.h"
#include "nlsar_split.h"
#include "nlsar_split3.cuh"
#include "nlsar_words.cuh"

namespace dcl {

namespace {

constexpr int kSimLeft = 8;  // similarity columns left of word column 0 (the halo lanes of a warp)

// ---- similarities -------------------------------------------------------------

constexpr int kSimTH = 16, kSimThreads = 256;

__host__ __device__ inline size_t sim3_smem(int wsh) { return (size_t)(kSimTH + wsh) * (32 + 2 * wsh) * 40; }

// One block: 32 x 16 pixels of the volume, two per thread (8 rows apart), the
// offsets z, z + Z, ..  The nine reals and ln det of a staged pixel are two
// float4 and one float2 plane; lanes read consecutive pixels.
// EXACT: with the arithmetic of nlsar3_kernel (nlsar_dim3.cu).
template <bool EXACT>
__global__ void __launch_bounds__(kSimThreads, 3)
    sim3_kernel(const float* __restrict__ s9, const float* __restrict__ ld, int Hp, int Wp, int pitch, size_t plane,
                int wsh, float c2d, int fy0, int fx0, float* __restrict__ sims, int srows, int spitch) {
  extern __shared__ float4 smem4[];
  const int RW = 32 + 2 * wsh, RH = kSimTH + wsh, RN = RW * RH;
  float4* sA = smem4;
  float4* sB = sA + RN;
  float2* sC = reinterpret_cast<float2*>(sB + RN);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.y * kSimTH, c0 = blockIdx.x * 32;
  // coordinates are clamped to the frame: the pixels a used weight needs are
  // inside it
  for (int r = warp; r < RH; r += kSimThreads / 32) {
    const size_t row = (size_t)min(max(fy0 + r0 + r, 0), Hp - 1) * pitch;
    for (int c = lane; c < RW; c += 32) {
      const size_t g = row + min(max(fx0 + c0 + c - wsh, 0), Wp - 1);
      float v[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) v[q] = s9[q * plane + g];
      const int i = r * RW + c;
      sA[i] = make_float4(v[0], v[1], v[2], v[3]);
      sB[i] = make_float4(v[4], v[5], v[6], v[7]);
      sC[i] = make_float2(v[8], ld[g]);
    }
  }
  __syncthreads();
  const int ci = warp * RW + lane + wsh;
  float4 a[2], b[2];
  float2 c[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    a[p] = sA[ci + 8 * p * RW];
    b[p] = sB[ci + 8 * p * RW];
    c[p] = sC[ci + 8 * p * RW];
  }
  const int sws = 2 * wsh + 1, nhalf = (sws * sws - 1) / 2;
  const bool in_c = c0 + lane < spitch;
  float* out = sims + (size_t)(r0 + warp) * spitch + c0 + lane;
  const size_t splane = (size_t)srows * spitch;
  for (int u = blockIdx.z; u < nhalf; u += gridDim.z) {
    const int v = u + wsh + 1;
    const int dy = v / sws, dx = v - dy * sws - wsh;
    const int ni = ci + dy * RW + dx;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float4 na = sA[ni + 8 * p * RW], nb = sB[ni + 8 * p * RW];
      const float2 nc = sC[ni + 8 * p * RW];
      const float sum[9] = {a[p].x + na.x, a[p].y + na.y, a[p].z + na.z, a[p].w + na.w, b[p].x + nb.x,
                            b[p].y + nb.y, b[p].z + nb.z, b[p].w + nb.w, c[p].x + nc.x};
      float sim;
      if (EXACT) {  // a lower-half offset: neighbour first (copy_symm_weights.cl:66-74)
        sim = -(((c2d + nc.y) + c[p].y) - 2.0f * logf(det3f(sum)));
      } else {
        const float t = (c[p].y + nc.y) + c2d;
        sim = fmaf(2.0f * 0.69314718f, __log2f(det3f(sum)), -t);
      }
      if (sim != sim) sim = 0.0f;
      if (in_c && r0 + warp + 8 * p < srows) out[u * splane + (size_t)(8 * p) * spitch] = sim;
    }
  }
}

// ---- weight codes -------------------------------------------------------------

constexpr int kWordsWarps = 8;

// One warp: a strip of VC columns x R rows of a pass's words for one offset.
// Similarity row 0 is the words' row 0 less the call's largest patch half
// `halo`.
template <int PH0, int PH1, int PH2, bool EXACT>
__global__ void __launch_bounds__(32 * kWordsWarps, 2)
    words3_kernel(const __grid_constant__ FilterParams P, int ps, const float* __restrict__ sims, int srows, int spitch,
                  int halo, char* __restrict__ words, int rows, int pitch, int R, int nbx, int items) {
  using Walk = WordWalk<PH0, PH1, PH2, EXACT>;
  using Word = typename WordOf<Walk::NP>::T;
  constexpr int PHM = Walk::PHM;
  const int lane = threadIdx.x & 31;
  const int item = blockIdx.x * kWordsWarps + (threadIdx.x >> 5);
  const int u = blockIdx.y;
  if (item >= items) return;
  const int by = item / nbx, bx = item - by * nbx;
  const int r0 = by * R, n = min(R, rows - r0);
  const int c = Walk::VC * bx + 4 * (lane - Walk::HL);
  const bool reads = c + kSimLeft + 4 <= spitch, writes = lane >= Walk::HL && lane < 32 - Walk::HL && c < pitch;
  const float4* in = reinterpret_cast<const float4*>(sims + ((size_t)u * srows + r0 + halo - PHM) * spitch + c +
                                                     kSimLeft);
  Word* out = reinterpret_cast<Word*>(words) + ((size_t)u * rows + r0) * pitch + c;
  Walk walk;
  walk.set(P, P.pass[ps], false);
  walk.start();
  const int step = spitch / 4;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int D = 3;  // rows in flight
  float4 nx[D];
#pragma unroll
  for (int k = 0; k < D; ++k) nx[k] = reads && k < n + 2 * PHM ? __ldcs(in + k * step) : zero;
  in += D * step;
  for (int i = 0; i < n + 2 * PHM; ++i) {
    const float4 v = nx[0];
#pragma unroll
    for (int k = 0; k + 1 < D; ++k) nx[k] = nx[k + 1];
    nx[D - 1] = reads && i + D < n + 2 * PHM ? __ldcs(in) : zero;
    in += step;
    float s[4 + 2 * PHM];
    s[PHM] = v.x;
    s[PHM + 1] = v.y;
    s[PHM + 2] = v.z;
    s[PHM + 3] = v.w;
    uint32_t w[4];
    walk.template row<false>(s, w);
    if (i >= 2 * PHM) {
      if (writes) store_words<Walk::NP>(out, w);
      out += pitch;
    }
  }
}

// ---- means --------------------------------------------------------------------

// One block: a 32 x TH tile, one pixel per thread, one row per warp; the 18
// planes of the tile and its window halo in four float4 planes and one float2
// plane (22 shared-memory wavefronts per pixel, offset and scale with three
// patch sizes are what bounds it).  Tables as in nlsar_split.cu, the third in
// 128-byte entries.
template <int WSH_, int TH_, int NPX_>
struct Mean3L {
  static constexpr int WSH = WSH_, TH = TH_, NPX = NPX_;
  static constexpr int WARPS = TH, THREADS = 32 * WARPS;
  static constexpr int SWS = 2 * WSH + 1;
  static constexpr int RO = 32 + 2 * WSH, ROH = TH + 2 * WSH, PLANE = RO * ROH;
  static constexpr int OFF_T2 = 256 * 256, OFF_CO = OFF_T2 + (NPX > 2 ? 256 * 128 : 0);  // bytes
  static constexpr int OFF_ONE = OFF_CO + PLANE * 72;
  static constexpr int BYTES = OFF_ONE + 16;
  static_assert(BYTES <= 227 * 1024, "shared memory");
};

struct Best3x {
  float e, a, s0, m[18];
  int rank, combo;
};

template <class L, int NP>
__device__ __forceinline__ void mean3_pass(const FilterParams& P, int ps, const char* __restrict__ pass_words, int rows,
                                           int wpitch, uint32_t lane_off, Best3x& best) {
  using Word = typename WordOf<NP>::T;
  constexpr int SWS = L::SWS, WSH = L::WSH, RO = L::RO, K = SWS;
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  const PassParams& pp = P.pass[ps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();  // the previous pass's tables are no longer read
  for (int i = tid; i < NP * 256 * 8; i += L::THREADS) {
    const int j = i >> 11, e = (i >> 3) & 255;
    const float w = e == kZeroCode ? 0.0f : P.wtab[pp.combo[j] * kMaxLut + e];
    const int at = j < 2 ? e * 256 + j * 128 : L::OFF_T2 + e * 128;
    *reinterpret_cast<float4*>(sm + at + (i & 7) * 16) = make_float4(w, w, w, w);
  }
  __syncthreads();
  float sw[NP], sww[NP], si2[NP];  // sum w, w^2, w I2^2
  float2 si01[NP], acc[NP][9];     // sums of w (I0^2, I1^2) and of w times the planes, in pairs
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    sw[j] = sww[j] = si2[j] = 0.0f;
    si01[j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int a = 0; a < 9; ++a) acc[j][a] = make_float2(0.f, 0.f);
  }
  const uint32_t lane4 = 4u * lane;
  auto weight = [&](uint32_t w, int j) {
    if (j == 2) return *reinterpret_cast<const float*>(sm + L::OFF_T2 + (((w >> 9) & 0x7F80u) | lane4));
    return *reinterpret_cast<const float*>(sm + j * 128 + __byte_perm(w, lane4, 0x5504 | (j << 4)));
  };
  const float4* tile = reinterpret_cast<const float4*>(sm + L::OFF_CO);
  const float2* tile2 = reinterpret_cast<const float2*>(tile + 4 * L::PLANE);
  auto accumulate = [&](const float (&w)[NP], int i) {
    float2 v[9];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 t = tile[q * L::PLANE + i];
      v[2 * q] = make_float2(t.x, t.y);
      v[2 * q + 1] = make_float2(t.z, t.w);
    }
    v[8] = tile2[i];
    // diagonal planes 0, 8, 16
    const float2 i01 = make_float2(__fmul_rn(v[0].x, v[0].x), __fmul_rn(v[4].x, v[4].x));
    const float i2 = __fmul_rn(v[8].x, v[8].x);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const float2 ww = make_float2(w[j], w[j]);
      sw[j] = __fadd_rn(sw[j], w[j]);
      sww[j] = __fmaf_rn(w[j], w[j], sww[j]);
      si01[j] = __ffma2_rn(ww, i01, si01[j]);
      si2[j] = __fmaf_rn(w[j], i2, si2[j]);
#pragma unroll
      for (int a = 0; a < 9; ++a) acc[j][a] = __ffma2_rn(ww, v[a], acc[j][a]);
    }
  };
  // words and their order as in nlsar_split.cu, a window row per run
  const uint32_t plane = (uint32_t)rows * wpitch;
  const Word* words = reinterpret_cast<const Word*>(pass_words);
  uint32_t off = lane_off + (uint32_t)(P.n_off / 2 - 1) * plane - (uint32_t)WSH * wpitch - (uint32_t)WSH;
  uint32_t step = 1u - plane;
  uint32_t buf[K];
  auto load = [&](int k) {
    buf[k] = __ldcg(words + off);
    off += step;
  };
#pragma unroll
  for (int k = 0; k < K; ++k) load(k);
  off += (uint32_t)wpitch - SWS;
  int ti = warp * RO + lane;
  for (int run = 0; run < SWS; ++run) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float w[NP];
      if (k == K / 2 && run == WSH) {
        // the centre: weight 1, read from memory so that w I^2 is rounded
        // before it is added, as for every other offset
        const float one = *reinterpret_cast<const float*>(sm + L::OFF_ONE);
#pragma unroll
        for (int j = 0; j < NP; ++j) w[j] = one;
      } else {
#pragma unroll
        for (int j = 0; j < NP; ++j) w[j] = weight(buf[k], j);
      }
      if (k == K / 2 && run + 1 == WSH) {
        off = lane_off;  // the next run's centre has no word; its lower half starts at word 0
        step = plane;
      } else if (run + 1 < SWS) {
        load(k);
      }
      accumulate(w, ti + k);
    }
    ti += RO;
    if (run + 1 < WSH) off += (uint32_t)wpitch - SWS;
  }
  // statistics over the three diagonal intensities, alpha, ENL', selection
  // (compute_nl_statistics.cl:92-101, compute_alphas.cl:30-41,
  // compute_enls_nobias.cl:19-22, best_params.cpp)
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const float s0 = sw[j], s1 = sww[j];
    const float enl = s0 * s0 / s1;
    float alpha = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float in = (d == 0 ? acc[j][0].x : (d == 1 ? acc[j][4].x : acc[j][8].x)) / s0;
      const float m2 = (d == 0 ? si01[j].x : (d == 1 ? si01[j].y : si2[j])) / s0;
      const float var = __fmaf_rn(-in, in, m2), num = __fmaf_rn(-in, in, var);
      alpha = fmaxf(alpha, fmaxf(0.0f, num / var));
    }
    if (P.alpha_zero) alpha = 0.0f;
    const float oma = 1.0f - alpha;
    const float enb = enl / (oma * oma + (alpha * alpha + 2.0f * alpha * (1.0f - alpha) / s0) * enl);
    const int combo = pp.combo[j];
    const int rank = P.combo[combo].rank;
    const bool take = (P.select_mode == 0) || (enb > best.e) || (enb == best.e && rank < best.rank);
    const bool take_fb = !take && best.combo < 0 && combo == P.fallback_combo;
    if (take) {
      best.e = enb;
      best.rank = rank;
    }
    if (take || take_fb) {
      best.combo = combo;
      best.a = alpha;
      best.s0 = s0;
#pragma unroll
      for (int a = 0; a < 9; ++a) {
        best.m[2 * a] = acc[j][a].x;
        best.m[2 * a + 1] = acc[j][a].y;
      }
    }
  }
}

struct WordOffsets {
  size_t at[kMaxPasses];  // byte offset of each pass's words in the volume
};

// A segment: the virtual rows filtered and the first column, its rows of words
// and words per row (the first is row vy0 - wsh, column vx0 - wsh), mean tiles
// per row.
struct Seg3 {
  int vy0, vy1, vx0;
  int rows, pitch, tiles_x;
};

// (the members of Seg3 one by one: with the struct as an argument the 12-row
// variant spills 256 bytes a thread instead of 12)
template <class L>
__global__ void __launch_bounds__(L::THREADS, 1)
    mean3_kernel(const __grid_constant__ FilterParams P, const __grid_constant__ Scene3 S, int Hp,
                 const char* __restrict__ vol, const __grid_constant__ WordOffsets wo, int vy0s, int vy1, int vx0s,
                 int rows, int wpitch, int tiles_x) {
  constexpr int WSH = L::WSH, RO = L::RO;
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = blockIdx.x / tiles_x, tx = blockIdx.x - ty * tiles_x;
  const int vy0 = vy0s + ty * L::TH, vx0 = vx0s + tx * 32;
  float4* tile = reinterpret_cast<float4*>(sm + L::OFF_CO);
  float2* tile2 = reinterpret_cast<float2*>(tile + 4 * L::PLANE);
  for (int r = warp; r < L::ROH; r += L::WARPS) {
    // rows past the frame are clamped (outputs that exist never use them)
    const size_t row = (size_t)min(vy0 - WSH + P.G + r, Hp - 1) * S.pitch + (vx0 - WSH + P.G);
    for (int c = lane; c < RO; c += 32) {
      const float* g = S.c18 + row + c;
      const int i = r * RO + c;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        tile[q * L::PLANE + i] = make_float4(g[(4 * q) * S.plane], g[(4 * q + 1) * S.plane], g[(4 * q + 2) * S.plane],
                                             g[(4 * q + 3) * S.plane]);
      tile2[i] = make_float2(g[16 * S.plane], g[17 * S.plane]);
    }
  }
  if (tid == 0) *reinterpret_cast<float*>(sm + L::OFF_ONE) = 1.0f;
  // pixels past the segment's last row and the last virtual column repeat it:
  // their words exist (columns are cut between tiles)
  const uint32_t lane_off = (uint32_t)(min(vy0 + warp, vy1 - 1) - vy0s + WSH) * wpitch +
                            (uint32_t)(min(vx0 + lane, S.vW) - vx0s) + WSH;
  Best3x best;
  best.e = -1.0f;
  best.a = 0.0f;
  best.s0 = 1.0f;
  best.rank = 0x7fffffff;
  best.combo = -1;
#pragma unroll
  for (int p = 0; p < 18; ++p) best.m[p] = 0.0f;
  for (int ps = 0; ps < P.npass; ++ps) {
    const char* w = vol + wo.at[ps];
    if constexpr (L::NPX == 1) {
      mean3_pass<L, 1>(P, ps, w, rows, wpitch, lane_off, best);
    } else if (P.pass[ps].np == 2) {
      mean3_pass<L, 2>(P, ps, w, rows, wpitch, lane_off, best);
    } else {
      mean3_pass<L, 3>(P, ps, w, rows, wpitch, lane_off, best);
    }
  }
  // blend with the centre (weighted_means.cl:79)
  const int vy = vy0 + warp, vx = vx0 + lane;
  const int oy = (vy < S.H - 1) ? vy : (vy == S.vH ? S.H - 1 : -1);
  const int ox = (vx < S.W - 1) ? vx : (vx == S.vW ? S.W - 1 : -1);
  if (oy < 0 || ox < 0 || vy >= vy1) return;
  const size_t n = (size_t)S.H * S.W, o = (size_t)oy * S.W + ox;
  const int ci = (warp + WSH) * RO + lane + WSH;
  const float oma = 1.0f - best.a;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    float2 cp;
    if (q == 8) {
      cp = tile2[ci];
    } else {
      const float4 t = tile[(q / 2) * L::PLANE + ci];
      cp = q & 1 ? make_float2(t.z, t.w) : make_float2(t.x, t.y);
    }
    S.out[(2 * q) * n + o] = oma * best.m[2 * q] / best.s0 + best.a * cp.x;
    S.out[(2 * q + 1) * n + o] = oma * best.m[2 * q + 1] / best.s0 + best.a * cp.y;
  }
}

// Means as nlsar3_kernel sums them, any window: the offsets in pairs, the upper
// half's first and its mirror after it, the centre last.  Tile, tables and
// staged planes as above, the window at run time.
__host__ __device__ constexpr int exact3_tables(int npx) { return 256 * 256 + (npx > 2 ? 256 * 128 : 0); }
inline size_t exact3_smem(int wsh, int th, int npx) {
  return exact3_tables(npx) + (size_t)(32 + 2 * wsh) * (th + 2 * wsh) * 72;
}
constexpr int kPairs3 = 4;  // offset pairs whose words are in flight

template <int TH, int NPX, int NP>
__device__ __forceinline__ void exact3_pass(const FilterParams& P, int ps, const char* __restrict__ pass_words,
                                            int rows, int wpitch, uint32_t lane_off, int RO, int PLANE,
                                            Best3x& best) {
  using Word = typename WordOf<NP>::T;
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  const PassParams& pp = P.pass[ps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wsh = P.wsh;
  __syncthreads();  // the previous pass's tables are no longer read
  for (int i = tid; i < NP * 256 * 8; i += 32 * TH) {
    const int j = i >> 11, e = (i >> 3) & 255;
    const float w = e == kZeroCode ? 0.0f : P.wtab[pp.combo[j] * kMaxLut + e];
    const int at = j < 2 ? e * 256 + j * 128 : 65536 + e * 128;
    *reinterpret_cast<float4*>(sm + at + (i & 7) * 16) = make_float4(w, w, w, w);
  }
  __syncthreads();
  float A[NP][5], m[NP][18];  // sum w, w^2, w I_d^2; of w times the planes
#pragma unroll
  for (int j = 0; j < NP; ++j) {
#pragma unroll
    for (int a = 0; a < 5; ++a) A[j][a] = 0.0f;
#pragma unroll
    for (int a = 0; a < 18; ++a) m[j][a] = 0.0f;
  }
  const uint32_t lane4 = 4u * lane;
  const float4* tile = reinterpret_cast<const float4*>(sm + exact3_tables(NPX));
  const float2* tile2 = reinterpret_cast<const float2*>(tile + 4 * PLANE);
  auto planes = [&](int i, float (&v)[18]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 t = tile[q * PLANE + i];
      v[4 * q] = t.x;
      v[4 * q + 1] = t.y;
      v[4 * q + 2] = t.z;
      v[4 * q + 3] = t.w;
    }
    const float2 t = tile2[i];
    v[16] = t.x;
    v[17] = t.y;
  };
  auto accumulate = [&](uint32_t word, int i) {
    float v[18], i2[3];
    planes(i, v);
#pragma unroll
    for (int d = 0; d < 3; ++d) i2[d] = __fmul_rn(v[diag_plane(d)], v[diag_plane(d)]);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int at = j == 2 ? 65536 + (int)(((word >> 9) & 0x7F80u) | lane4)
                            : j * 128 + (int)__byte_perm(word, lane4, 0x5504 | (j << 4));
      const float w = *reinterpret_cast<const float*>(sm + at);
      A[j][0] = __fadd_rn(A[j][0], w);
      A[j][1] = __fmaf_rn(w, w, A[j][1]);
#pragma unroll
      for (int q = 0; q < 3; ++q) A[j][2 + q] = __fmaf_rn(w, i2[q], A[j][2 + q]);
#pragma unroll
      for (int q = 0; q < 18; ++q) m[j][q] = __fmaf_rn(w, v[q], m[j][q]);
    }
  };
  // pairs and their words as in nlsar_split.cu
  const uint32_t plane = (uint32_t)rows * wpitch;
  const Word* words = reinterpret_cast<const Word*>(pass_words);
  const int nhalf = P.n_off / 2;
  uint32_t up[kPairs3], down[kPairs3];
  int li = nhalf - 1, ldy = wsh, ldx = wsh;  // next pair to load
  auto load = [&](int k) {
    if (li >= 0) {
      const uint32_t off = lane_off + (uint32_t)li * plane;
      down[k] = __ldcg(words + off);
      up[k] = __ldcg(words + (off - (uint32_t)(ldy * wpitch + ldx)));
      --li;
      if (--ldx < -wsh) ldx = wsh, --ldy;
    }
  };
#pragma unroll
  for (int k = 0; k < kPairs3; ++k) load(k);
  const int ci = (warp + wsh) * RO + lane + wsh;
  int d = wsh * RO + wsh, dx = wsh;  // place of x + o after x
  for (int i = nhalf - 1; i >= 0; i -= kPairs3) {
#pragma unroll
    for (int k = 0; k < kPairs3; ++k) {
      if (i - k < 0) break;
      const uint32_t wu = up[k], wd = down[k];
      load(k);
      accumulate(wu, ci - d);
      accumulate(wd, ci + d);
      --d;
      if (--dx < -wsh) dx = wsh, d -= RO - 2 * wsh - 1;
    }
  }
  // centre weight 1, statistics, alpha, ENL', selection (nlsar_dim3.cu)
  float c[18];
  planes(ci, c);
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const float s0 = A[j][0] + 1.0f, s1 = A[j][1] + 1.0f;
    const float enl = s0 * s0 / s1;
    float alpha = 0.0f;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float cd = c[diag_plane(q)];
      const float in = (m[j][diag_plane(q)] + cd) / s0;
      const float var = __fmaf_rn(cd, cd, A[j][2 + q]) / s0 - in * in;
      alpha = fmaxf(alpha, fmaxf(0.0f, (var - in * in) / var));
    }
    if (P.alpha_zero) alpha = 0.0f;
    const float oma = 1.0f - alpha;
    const float enb = enl / (oma * oma + (alpha * alpha + 2.0f * alpha * (1.0f - alpha) / s0) * enl);
    const int combo = pp.combo[j];
    const int rank = P.combo[combo].rank;
    const bool take = (P.select_mode == 0) || (enb > best.e) || (enb == best.e && rank < best.rank);
    const bool take_fb = !take && best.combo < 0 && combo == P.fallback_combo;
    if (take) {
      best.e = enb;
      best.rank = rank;
    }
    if (take || take_fb) {
      best.combo = combo;
      best.a = alpha;
      best.s0 = s0;
#pragma unroll
      for (int q = 0; q < 18; ++q) best.m[q] = m[j][q] + c[q];
    }
  }
}

template <int TH, int NPX>
__global__ void __launch_bounds__(32 * TH, 1)
    exact3_mean_kernel(const __grid_constant__ FilterParams P, const __grid_constant__ Scene3 S, int Hp,
                       const char* __restrict__ vol, const __grid_constant__ WordOffsets wo,
                       const __grid_constant__ Seg3 G) {
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wsh = P.wsh;
  const int RO = 32 + 2 * wsh, ROH = TH + 2 * wsh, PLANE = RO * ROH;
  const int ty = blockIdx.x / G.tiles_x, tx = blockIdx.x - ty * G.tiles_x;
  const int vy0 = G.vy0 + ty * TH, vx0 = G.vx0 + tx * 32;
  float4* tile = reinterpret_cast<float4*>(sm + exact3_tables(NPX));
  float2* tile2 = reinterpret_cast<float2*>(tile + 4 * PLANE);
  for (int r = warp; r < ROH; r += TH) {
    const size_t row = (size_t)min(vy0 - wsh + P.G + r, Hp - 1) * S.pitch + (vx0 - wsh + P.G);
    for (int c = lane; c < RO; c += 32) {
      const float* g = S.c18 + row + c;
      const int i = r * RO + c;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        tile[q * PLANE + i] = make_float4(g[(4 * q) * S.plane], g[(4 * q + 1) * S.plane], g[(4 * q + 2) * S.plane],
                                          g[(4 * q + 3) * S.plane]);
      tile2[i] = make_float2(g[16 * S.plane], g[17 * S.plane]);
    }
  }
  // pixels past the segment's last row and the last virtual column repeat it:
  // their words exist (columns are cut between tiles)
  const uint32_t lane_off = (uint32_t)(min(vy0 + warp, G.vy1 - 1) - G.vy0 + wsh) * G.pitch +
                            (uint32_t)(min(vx0 + lane, S.vW) - G.vx0) + wsh;
  Best3x best;
  best.e = -1.0f;
  best.a = 0.0f;
  best.s0 = 1.0f;
  best.rank = 0x7fffffff;
  best.combo = -1;
#pragma unroll
  for (int p = 0; p < 18; ++p) best.m[p] = 0.0f;
  for (int ps = 0; ps < P.npass; ++ps) {
    const char* w = vol + wo.at[ps];
    if constexpr (NPX == 1) {
      exact3_pass<TH, NPX, 1>(P, ps, w, G.rows, G.pitch, lane_off, RO, PLANE, best);
    } else if (P.pass[ps].np == 2) {
      exact3_pass<TH, NPX, 2>(P, ps, w, G.rows, G.pitch, lane_off, RO, PLANE, best);
    } else {
      exact3_pass<TH, NPX, 3>(P, ps, w, G.rows, G.pitch, lane_off, RO, PLANE, best);
    }
  }
  const int vy = vy0 + warp, vx = vx0 + lane;
  const int oy = (vy < S.H - 1) ? vy : (vy == S.vH ? S.H - 1 : -1);
  const int ox = (vx < S.W - 1) ? vx : (vx == S.vW ? S.W - 1 : -1);
  if (oy < 0 || ox < 0 || vy >= G.vy1) return;
  const size_t n = (size_t)S.H * S.W, o = (size_t)oy * S.W + ox;
  const int ci = (warp + wsh) * RO + lane + wsh;
  const float oma = 1.0f - best.a;
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    const float cp = q < 16 ? reinterpret_cast<const float*>(tile + (q / 4) * PLANE + ci)[q & 3]
                            : reinterpret_cast<const float*>(tile2 + ci)[q & 1];
    S.out[q * n + o] = oma * best.m[q] / best.s0 + best.a * cp;
  }
}

// ---- host ---------------------------------------------------------------------

constexpr int kTall3 = 12;  // rows of the tallest mean tile (segments hold whole tiles of 12 and 8)

size_t word_bytes(int np) { return np == 3 ? 4 : np; }
int div_up(int a, int b) { return (a + b - 1) / b; }

int mean_tiles(const Seg3& G, int th) { return G.tiles_x * div_up(G.vy1 - G.vy0, th); }

template <int TH, int NPX>
cudaError_t launch_mean3_t(const FilterParams& F, const Scene3& S, int Hp, const char* vol, const WordOffsets& wo,
                           const Seg3& G, cudaStream_t st) {
  using L = Mean3L<10, TH, NPX>;
  static size_t allowed[kMaxDevices];
  const cudaError_t e = allow_dynamic_smem((const void*)mean3_kernel<L>, L::BYTES, allowed);
  if (e != cudaSuccess) return e;
  mean3_kernel<L><<<mean_tiles(G, TH), L::THREADS, L::BYTES, st>>>(F, S, Hp, vol, wo, G.vy0, G.vy1, G.vx0, G.rows,
                                                                   G.pitch, G.tiles_x);
  return cudaGetLastError();
}

template <int NPX>
cudaError_t launch_mean3(int th, const FilterParams& F, const Scene3& S, int Hp, const char* vol,
                         const WordOffsets& wo, const Seg3& G, cudaStream_t st) {
  switch (th) {
    case 4: return launch_mean3_t<4, NPX>(F, S, Hp, vol, wo, G, st);
    case 8: return launch_mean3_t<8, NPX>(F, S, Hp, vol, wo, G, st);
    default: return launch_mean3_t<kTall3, NPX>(F, S, Hp, vol, wo, G, st);
  }
}

template <int TH, int NPX>
cudaError_t launch_exact3_t(const FilterParams& F, const Scene3& S, int Hp, const char* vol, const WordOffsets& wo,
                            const Seg3& G, cudaStream_t st) {
  static size_t allowed[kMaxDevices];
  const cudaError_t e = allow_dynamic_smem((const void*)exact3_mean_kernel<TH, NPX>, kSplitSmem, allowed);
  if (e != cudaSuccess) return e;
  exact3_mean_kernel<TH, NPX><<<mean_tiles(G, TH), 32 * TH, exact3_smem(F.wsh, TH, NPX), st>>>(F, S, Hp, vol, wo, G);
  return cudaGetLastError();
}

template <int NPX>
cudaError_t launch_exact3(int th, const FilterParams& F, const Scene3& S, int Hp, const char* vol,
                          const WordOffsets& wo, const Seg3& G, cudaStream_t st) {
  return th == 4 ? launch_exact3_t<4, NPX>(F, S, Hp, vol, wo, G, st)
                 : launch_exact3_t<8, NPX>(F, S, Hp, vol, wo, G, st);
}

template <int PH0, int PH1, int PH2, bool EXACT>
cudaError_t launch_words3(const FilterParams& F, int ps, const float* sims, int srows, int spitch, char* words,
                          int rows, int pitch, int sms, cudaStream_t st) {
  using Walk = WordWalk<PH0, PH1, PH2, EXACT>;
  const int nbx = div_up(pitch, Walk::VC);
  // strips of up to 64 rows (each walks 2 PHM more); shorter ones where that
  // leaves fewer than 16 warps per SM
  int R = 64;
  const int nhalf = F.n_off / 2;
  while (R > 8 && (long long)nbx * div_up(rows, R) * nhalf < 16LL * sms) R /= 2;
  const int items = nbx * div_up(rows, R);
  words3_kernel<PH0, PH1, PH2, EXACT><<<dim3(div_up(items, kWordsWarps), nhalf), 32 * kWordsWarps, 0, st>>>(
      F, ps, sims, srows, spitch, F.phm, words, rows, pitch, R, nbx, items);
  return cudaGetLastError();
}

// pass shapes: 0 {1,2,3}, 1 {4,5}, 2..6 the single halves 1..5, 7 {1,2}; -1 none
int pass_shape3(const PassParams& p) {
  if (p.np == 3 && p.ph[0] == 1 && p.ph[1] == 2 && p.ph[2] == 3) return 0;
  if (p.np == 2 && p.ph[0] == 4 && p.ph[1] == 5) return 1;
  if (p.np == 1 && p.ph[0] >= 1 && p.ph[0] <= 5) return 1 + p.ph[0];
  if (p.np == 2 && p.ph[0] == 1 && p.ph[1] == 2) return 7;
  return -1;
}

}  // namespace

Split3 split3_layout(const Plan& pl, const Scene3& S, size_t budget) {
  const FilterParams& F = pl.P;
  Split3 L;
  const int nhalf = F.n_off / 2;
  if (!split_tables_ok(pl) || F.npass < 1 || F.wsh < 1) return L;
  L.exact = !(pl.fast && fast3_supported(F));
  if (L.exact && (pl.generic_only || F.prec != 0)) return L;
  // the launches of three kernels outweigh eight offsets of a small scene:
  // 64 x 70 with search 3 takes 73 us (nlsar3_kernel 61), with search 5 75 us
  // (112), 280 x 290 with search 3 98 us (124)
  if (L.exact && F.wsh == 1 && (long long)S.H * S.W < 65536) return L;
  int np_min = kPatchPerPass, npx = 1;
  for (int i = 0; i < F.npass; ++i) {
    if (pass_shape3(F.pass[i]) < 0) return L;
    np_min = std::min(np_min, F.pass[i].np);
    npx = std::max(npx, F.pass[i].np);
  }
  // passes of one size come alone; the staged window has to fit
  if (npx > 1 && np_min == 1) return L;
  npx = npx > 1 ? 3 : 1;
  if (L.exact && (exact3_smem(F.wsh, 4, npx) > kSplitSmem || sim3_smem(F.wsh) > kSplitSmem)) return L;
  // a segment's rows of similarities and of words, and its volume; 32-bit word
  // offsets within a pass
  const int extra_s = F.wsh + 2 * F.phm, extra_w = F.wsh, width = S.vW + 1, total = S.vH + 1;
  auto pitch_of = [&](int cols) { return (cols + 2 * F.wsh + 15) / 16 * 16; };
  auto sims = [&](int rows, int cols) {
    return ((size_t)nhalf * (rows + extra_s) * (pitch_of(cols) + 2 * kSimLeft) * sizeof(float) + 255) / 256 * 256;
  };
  auto volume = [&](int rows, int cols) {
    size_t bytes = sims(rows, cols);
    for (int i = 0; i < F.npass; ++i)
      bytes += ((size_t)nhalf * (rows + extra_w) * pitch_of(cols) * word_bytes(F.pass[i].np) + 255) / 256 * 256;
    return bytes;
  };
  auto fits = [&](int rows, int cols) {
    return volume(rows, cols) <= budget && (size_t)nhalf * (rows + extra_w) * pitch_of(cols) <= 0x3fffffff;
  };
  // the largest multiple of `unit` up to `most` that fits, 0 for none
  auto largest = [&](int most, int unit, auto ok) {
    int lo = 0, hi = most / unit;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (ok(mid * unit)) lo = mid; else hi = mid - 1;
    }
    return lo * unit;
  };
  constexpr int unit = 2 * kTall3;  // whole tiles of 12 and 8 rows
  int cols = width, rows = largest(div_up(total, unit) * unit, unit, [&](int r) { return fits(r, width); });
  if (rows == 0) {
    rows = unit;
    cols = largest(div_up(width, 32) * 32, 32, [&](int c) { return fits(unit, c); });
    if (cols == 0) return L;
    cols = div_up(div_up(width, div_up(width, cols)), 32) * 32;
  }
  L.rows = div_up(div_up(total, div_up(total, rows)), unit) * unit;
  L.cols = cols;
  L.pitch = pitch_of(cols);
  L.spitch = L.pitch + 2 * kSimLeft;
  L.sim_bytes = sims(L.rows, cols);
  L.vol_bytes = volume(L.rows, cols);
  return L;
}

cudaError_t launch_split3(const Plan& pl, const FilterParams& F, const Scene3& S, int Hp, int Wp, const Split3& L,
                          char* vol, int vy0, int vy1, int vx0, int vx1, int sms, cudaStream_t st) {
  const int nhalf = F.n_off / 2;
  const int rows = vy1 - vy0 + F.wsh, srows = rows + 2 * F.phm;
  float* sims = reinterpret_cast<float*>(vol);
  WordOffsets wo;
  size_t at = L.sim_bytes;
  for (int i = 0; i < F.npass; ++i) {
    wo.at[i] = at;
    at += ((size_t)nhalf * rows * L.pitch * word_bytes(F.pass[i].np) + 255) / 256 * 256;
  }
  static size_t allowed[kMaxDevices];
  static size_t allowed_exact[kMaxDevices];
  cudaError_t e = L.exact ? allow_dynamic_smem((const void*)sim3_kernel<true>, kSplitSmem, allowed_exact)
                          : allow_dynamic_smem((const void*)sim3_kernel<false>, sim3_smem(F.wsh), allowed);
  if (e != cudaSuccess) return e;
  int slot = -1, npx = 1;
  for (int ps = 0; ps < F.npass; ++ps) {
    const PassParams& pp = F.pass[ps];
    npx = std::max(npx, pp.np);
    if (pp.scale_slot != slot) {
      slot = pp.scale_slot;
      // similarity row 0 is virtual row vy0 - wsh - phm, column 0 virtual
      // column vx0 - wsh - kSimLeft; offset groups fill four blocks per SM
      dim3 grid(div_up(L.spitch, 32), div_up(srows, kSimTH));
      grid.z = std::max(1, std::min(nhalf, div_up(4 * sms, (int)(grid.x * grid.y))));
      e = launch_kernel(L.exact ? sim3_kernel<true> : sim3_kernel<false>, grid, kSimThreads, sim3_smem(F.wsh), st,
                        S.s9[slot], S.ld[slot], Hp, Wp, S.pitch, S.plane, F.wsh, F.c2d, vy0 - F.wsh - F.phm + F.G,
                        vx0 + F.G - F.wsh - kSimLeft, sims, srows, L.spitch);
      profile_count(1);
      if (e != cudaSuccess) return e;
    }
    char* words = vol + wo.at[ps];
    auto codes = [&](auto launch) {
      return launch(F, ps, sims, srows, L.spitch, words, rows, L.pitch, sms, st);
    };
    auto shape = [&](auto exact) {
      constexpr bool EXACT = decltype(exact)::value;
      switch (pass_shape3(pp)) {
        case 0: return codes(launch_words3<1, 2, 3, EXACT>);
        case 1: return codes(launch_words3<4, 5, -1, EXACT>);
        case 2: return codes(launch_words3<1, -1, -1, EXACT>);
        case 3: return codes(launch_words3<2, -1, -1, EXACT>);
        case 4: return codes(launch_words3<3, -1, -1, EXACT>);
        case 5: return EXACT ? codes(launch_words3<4, -1, -1, true>) : cudaErrorInvalidValue;
        case 6: return EXACT ? codes(launch_words3<5, -1, -1, true>) : cudaErrorInvalidValue;
        default: return EXACT ? codes(launch_words3<1, 2, -1, true>) : cudaErrorInvalidValue;
      }
    };
    e = L.exact ? shape(std::true_type{}) : shape(std::false_type{});
    profile_count(1);
    if (e != cudaSuccess) return e;
  }
  // rows of the mean tiles: waves of blocks times a block's time
  const Seg3 G{vy0, vy1, vx0, rows, L.pitch, div_up(vx1 - vx0, 32)};
  int th = kTall3;
  double best = 0.0;
  for (int t : {kTall3, 8, 4}) {
    const double cost = (double)div_up(mean_tiles(G, t), sms) * (t == kTall3 ? 1.0 : (t == 8 ? 0.72 : 0.45));
    if (best == 0.0 || cost < 0.98 * best) {
      best = cost;
      th = t;
    }
  }
  profile_count(1);
  if (L.exact) {
    const int t = th == 4 || exact3_smem(F.wsh, 8, npx == 1 ? 1 : 3) > kSplitSmem ? 4 : 8;
    return npx == 1 ? launch_exact3<1>(t, F, S, Hp, vol, wo, G, st)
                    : launch_exact3<3>(t, F, S, Hp, vol, wo, G, st);
  }
  return npx == 1 ? launch_mean3<1>(th, F, S, Hp, vol, wo, G, st)
                  : launch_mean3<3>(th, F, S, Hp, vol, wo, G, st);
}

}  // namespace dcl

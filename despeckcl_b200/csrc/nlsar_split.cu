// NL-SAR in two kernels around a volume of weight indices, for sm_100a: the
// same results, bit for bit, as the fused tile kernel (nlsar_fast.cu), with
// every weight computed once.
//
// The weight of offset -o at pixel x is the weight of o at x - o
// (copy_symm_weights.cl:56-76; the similarity is symmetric in its two pixels,
// so both have the same bits), and a weight is one of at most 256 table
// entries or zero.  So:
//
//  nlsar_index_kernel  for the lower half window (dy > 0, or dy = 0 and
//      dx > 0), every scale and patch size: GLR similarity, patch sums and
//      the index of the composite weight (compute_weights.cl:40-51), one byte
//      per patch size; three patch sizes share a 32-bit word per (offset,
//      pixel).
//  nlsar_mean_kernel   per output pixel: for all offsets in the reference's
//      row-major order (compute_nl_statistics.cl:77-78) the word of o at x
//      (lower half) or at x + q for q = -o (upper half), the weights from the
//      tables, the accumulators, and after all passes the selection and the
//      blended output.
//
// The fused kernel computes every weight twice (once per direction) on tiles
// whose patch halo costs 1.41x, and moves similarities and horizontal sums
// through shared memory three times with two block barriers per three offsets
// (125.7 thread instructions per pixel, offset and scale).  Here the index
// kernel has no accumulators, so it can hold the vertical sums of a column in
// registers: one warp walks down 128 columns for one offset with no barrier.
//
// Settings without a specialised fused kernel (other windows, patches {3,5})
// take the same way with the arithmetic and summation order of nlsar_kernels.cu
// (EXACT, nlsar_exact_mean_kernel), whose results they give bit for bit.
//
// The volume of one pass is (sws^2 - 1) / 2 words of 1, 2 or 4 bytes per pixel
// (220 to 880 B at search 21), so a scene is filtered in segments whose volume
// fits a budget (kSplitBudgetBytes), index kernel and mean kernel in turn: runs
// of whole rows, cut in columns where one row of tiles is too much (kept as
// long as they can be: every segment works out wsh more rows of codes).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "dcl_internal.h"
#include "nlsar_math.cuh"
#include "nlsar_split.h"
#include "nlsar_words.cuh"

namespace dcl {

namespace {

constexpr int kIdxWarps = 16;
constexpr int kIdxThreads = 32 * kIdxWarps;
constexpr int kIdxLoads = 6;  // pixels a lane stages of a row

__host__ __device__ inline int idx_left(int wsh) { return (wsh + 3) / 4 * 4; }  // staged columns left of lane 0
// float4 slots of a staged row: five per four pixels (see the kernel)
__host__ __device__ inline int idx_row_slots(int wsh) { return 5 * ((idx_left(wsh) + 128 + wsh + 3) / 4); }
__host__ __device__ inline size_t idx_smem(int wsh, int phm, int R) {
  return (size_t)(R + 2 * phm + wsh) * idx_row_slots(wsh) * 20;
}

// The similarity of a lower-half offset as nlsar_kernels.cu evaluates it
// (neighbour first, copy_symm_weights.cl:66-74; a NaN counts as 0 in WordWalk)
__device__ __forceinline__ float glr_lower(float c2d, const float4 a, float la, const float4 b, float lb) {
  const float s00 = a.x + b.x, s11 = a.y + b.y, sre = a.z + b.z, sim = a.w + b.w;
  const float det = (s00 * s11) - (sre * sre + sim * sim);
  return -(((c2d + lb) + la) - 2.0f * logf(det));
}

// One block: a rectangle of R rows x VC columns of one segment's volume, one
// pass, the offsets u = 16 z + warp, 16 (z + Z) + warp, ...
//
// Staged in shared memory: the scaled covariance of the rectangle with its
// patch halo and the half window's halo (rows below, columns both sides).
// Every fourth pixel is followed by a slot that holds the four pixels' 1/(4
// det): a lane's four columns are five slots apart from the next lane's, so
// the 16-byte loads of eight lanes fall in distinct bank groups for every
// offset, and the centre's four determinants come in one load.  A second
// plane with the same indexing holds 1/(4 det) alone for the neighbours
// (4-byte loads, five words apart: conflict free).
//
// A warp walks down the rows for one offset (WordWalk), a lane evaluating the
// four similarities of its columns per row.
//
// EXACT: the arithmetic of nlsar_kernels.cu for the settings that it serves:
// the staged term is ln det from the frame, the similarity takes the rounded
// logarithm, the index a rounded division.
template <int PH0, int PH1, int PH2, bool EXACT>
__global__ void __launch_bounds__(kIdxThreads, 1)
    nlsar_index_kernel(const __grid_constant__ FilterParams P, const SceneDesc* __restrict__ scenes,
                       const SplitSeg* __restrict__ segs, int nseg, const __grid_constant__ PassList passes,
                       int shape, char* __restrict__ vol) {
  using Walk = WordWalk<PH0, PH1, PH2, EXACT>;
  constexpr int NP = Walk::NP, PHM = Walk::PHM, HL = Walk::HL, VC = Walk::VC;
  using Word = typename WordOf<NP>::T;
  extern __shared__ float4 smem4[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].idx_begin[shape] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const SplitSeg& S = segs[lo];
  const SceneDesc& D = scenes[S.scene];
  const int ps = passes.id[blockIdx.z];
  const PassParams& pp = P.pass[ps];
  const int bx_n = S.idx_bx[shape];
  const int lb = (int)blockIdx.x - S.idx_begin[shape];
  const int by = lb / bx_n, bx = lb - by * bx_n;
  const int wsh = P.wsh, sws = P.sws, left = idx_left(wsh), SP = idx_row_slots(wsh);
  const int r0 = by * S.idx_R[shape];                      // first volume row of the block
  const int R = min(S.idx_R[shape], S.rows - r0);
  const int nrow = R + 2 * PHM + wsh;               // staged rows
  float4* sC = smem4;
  float* sL = reinterpret_cast<float*>(smem4 + nrow * SP);
  {
    // staged column 0 is `left` columns before lane 0's first; volume column
    // c is virtual column vx0 + c - wsh.  Coordinates are clamped to the frame:
    // the pixels a used weight needs are inside it.
    const int Hp = D.tiles_y * P.tile_h + 2 * P.G, Wp = D.tiles_x * kTileW + 2 * P.G;
    const int fx0 = S.vx0 + VC * bx - 4 * HL - wsh - left + P.G, fy0 = S.row0 + r0 - PHM + P.G;
    const int ncol = left + 128 + wsh;
    const float4* cs = D.cs[pp.scale_slot];
    const float* ld = D.ld[pp.scale_slot];
    constexpr int U = kIdxLoads;  // ncol <= 32 U (split_supported), up to search 65
    for (int r = warp; r < nrow; r += kIdxWarps) {
      const size_t row = (size_t)min(max(fy0 + r, 0), Hp - 1) * D.pitch;
      float4 v[U];
      float term[U];
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (lane + 32 * k < ncol) {
          const size_t g = row + min(max(fx0 + lane + 32 * k, 0), Wp - 1);
          v[k] = cs[g];
          if (EXACT) term[k] = ld[g];
        }
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int p = lane + 32 * k;
        if (p < ncol) {
          const int slot = r * SP + p + (p >> 2);
          const float t = EXACT ? term[k] : pixel_term<kPrecRatio>(v[k]);
          sC[slot] = v[k];
          sL[slot] = t;
          reinterpret_cast<float*>(sC + r * SP + 5 * (p >> 2) + 4)[p & 3] = t;
        }
      }
    }
  }
  Walk walk;
  walk.set(P, pp, !EXACT);  // patch sums in log2 units (nlsar_fast.cu)
  __syncthreads();

  const int nhalf = P.n_off / 2;
  const int c = VC * bx + 4 * (lane - HL);  // this lane's first volume column
  const bool writes = lane >= HL && lane < 32 - HL && c < S.pitch;
  const size_t plane = (size_t)S.rows * S.pitch;
  Word* out0 = reinterpret_cast<Word*>(vol + S.vol + S.pass[ps]) + (ptrdiff_t)r0 * S.pitch + c;

  for (int u = (int)blockIdx.y * kIdxWarps + warp; u < nhalf; u += kIdxWarps * (int)gridDim.y) {
    // lower half window, row-major: (0, 1) .. (0, wsh), (1, -wsh) ..
    const int v = u + wsh + 1;
    const int dy = v / sws, dx = v - dy * sws - wsh;
    // neighbour of column j: pixel t + j of the staged row, t = left + dx plus
    // four per lane; M = t mod 4 fixes the slots of all four relative to the
    // first's
    const int t0 = left + dx;
    Word* out = out0 + (size_t)u * plane;
    const float4* ctr = sC + 5 * (lane + (left >> 2));
    const int n0 = dy * SP + 5 * (lane + (t0 >> 2)) + (t0 & 3);
    auto down = [&](auto m_tag) {
      constexpr int M = decltype(m_tag)::value;
      const float4* nbr = sC + n0;
      const float* nld = sL + n0;
      walk.start();
      for (int i = 0; i < R + 2 * PHM; ++i) {
        float s[4 + 2 * PHM];
        const float4 la = ctr[4];
        const float la4[4] = {la.x, la.y, la.z, la.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = j + (M + j >= 4 ? 1 : 0);
          s[PHM + j] = EXACT ? glr_lower(P.c2d, ctr[j], la4[j], nbr[n], nld[n]) : glr_ratio(ctr[j], la4[j], nbr[n], nld[n]);
        }
        ctr += SP;
        nbr += SP;
        nld += SP;
        uint32_t w[4];
        walk.template row<true>(s, w);
        if (i >= 2 * PHM) {
          if (writes) store_words<NP>(out, w);
          out += S.pitch;
        }
      }
    };
    switch (t0 & 3) {
      case 0: down(std::integral_constant<int, 0>{}); break;
      case 1: down(std::integral_constant<int, 1>{}); break;
      case 2: down(std::integral_constant<int, 2>{}); break;
      default: down(std::integral_constant<int, 3>{});
    }
  }
}

// ---------------------------------------------------------------------------
// mean kernel
// ---------------------------------------------------------------------------

// One block: a 32 x TH tile of outputs, one pixel per thread, one row per
// warp.  Of the accumulators that share a weight, six (ten with 8-plane input)
// are updated two per packed (f32x2) FMA.  Bound by issue slots (about 35 per
// pixel, offset and scale) and FMA cycles (packed FMAs take two) in about
// equal parts; measured and slower at 4096^2 (40.7 ms): two pixels per thread
// in 16 warps (42.4), two scales per sweep with patch sizes packed in pairs
// (42.9), the words through a TMA ring (48.5: one thread's issue sets the
// pace).
//
// Weight tables: one copy per lane, so the gathers have no bank conflicts.
// Tables 0 and 1 interleave in 256-byte entries and table 2 has them to
// itself, so one byte permute of the word and 4 lane gives an entry's byte
// offset.
template <int WSH_, int TH_, bool FULL8_, int NPX_>
struct MeanL {
  static constexpr int WSH = WSH_, TH = TH_, NPX = NPX_;  // NPX: patch sizes of the largest pass
  static constexpr bool FULL8 = FULL8_;
  static constexpr int WARPS = TH, THREADS = 32 * WARPS;
  static constexpr int NA = FULL8 ? 12 : 8, NM = FULL8 ? 8 : 4;
  static constexpr int SWS = 2 * WSH + 1;
  // window columns per run, the words in flight ahead: 32 warps hide their
  // latency with 7, fewer warps want a whole window row (1024^2 in 16-row
  // tiles: 2.86 ms with 7, 2.68 with 21)
  static constexpr int K = TH > 16 ? 7 : 21;
  static constexpr int RUNS = SWS * SWS / K, MID = RUNS / 2, ROWRUNS = SWS / K;
  static constexpr int RO = 32 + 2 * WSH, ROH = TH + 2 * WSH;  // staged covariance
  static constexpr int PLANE = RO * ROH;                        // float4 per staged plane
  static constexpr int NPL = FULL8 ? 2 : 1;
  static constexpr int OFF_CO = (NPX + 1) / 2 * 256 * 256;      // bytes, after the tables
  static constexpr int OFF_ONE = OFF_CO + NPL * PLANE * 16;
  static constexpr int BYTES = OFF_ONE + 16;
  static_assert(SWS % K == 0 && K > WSH % K, "runs tile a window row");
  static_assert(ROWRUNS % 2 == 1 && K % 2 == 1, "the centre is the middle of the middle run");
  static_assert(BYTES <= 227 * 1024, "shared memory");
};

// One pass of NP patch sizes over the window.  lane_off: the word of the
// thread's pixel in a plane of the volume.
template <class L, int NP>
__device__ __forceinline__ void mean_pass(const FilterParams& P, int ps, const char* __restrict__ vol,
                                          const SplitSeg& G, uint32_t lane_off, Best<1, L::NM>& best) {
  using Word = typename WordOf<NP>::T;
  constexpr int NA = L::NA, K = L::K, SWS = L::SWS, WSH = L::WSH, RO = L::RO;
  static_assert(NP <= L::NPX, "tables");
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  const PassParams& pp = P.pass[ps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __syncthreads();  // the previous pass's tables are no longer read
  for (int i = tid; i < NP * 256 * 8; i += L::THREADS) {
    const int m = i >> 11, e = (i >> 3) & 255;
    const float w = e == kZeroCode ? 0.0f : P.wtab[pp.combo[m] * kMaxLut + e];
    *reinterpret_cast<float4*>(sm + (m >> 1) * 65536 + e * 256 + (m & 1) * 128 + (i & 7) * 16) =
        make_float4(w, w, w, w);
  }
  __syncthreads();
  float sw[NP], sww[NP];        // sum w, sum w^2
  float2 acc[NP][NA / 2 - 1];  // sums of w (I0, I1), w (I0^2, I1^2), w C01, 8-plane input's other four
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    sw[j] = sww[j] = 0.0f;
#pragma unroll
    for (int a = 0; a < NA / 2 - 1; ++a) acc[j][a] = make_float2(0.f, 0.f);
  }
  const uint32_t lane4 = 4u * lane;
  auto weight = [&](uint32_t w, int j) {
    return *reinterpret_cast<const float*>(sm + (j >> 1) * 65536 + (j & 1) * 128 +
                                           __byte_perm(w, lane4, 0x5504 | (j << 4)));
  };
  // each component of a packed operation is rounded like the scalar add /
  // multiply / fma
  auto accumulate = [&](const float (&w)[NP], const float4* v) {
    const float4 a = v[0];
    const float2 i01 = make_float2(a.x, a.y), c01 = make_float2(a.z, a.w);
    const float2 sq = __fmul2_rn(i01, i01);
    float2 ex[2];
    if constexpr (L::FULL8) {
      const float4 e = v[L::PLANE];
      ex[0] = make_float2(e.x, e.y);
      ex[1] = make_float2(e.z, e.w);
    }
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const float2 ww = make_float2(w[j], w[j]);
      sw[j] = __fadd_rn(sw[j], w[j]);
      sww[j] = __fmaf_rn(w[j], w[j], sww[j]);
      acc[j][0] = __ffma2_rn(ww, i01, acc[j][0]);
      acc[j][1] = __ffma2_rn(ww, sq, acc[j][1]);
      acc[j][2] = __ffma2_rn(ww, c01, acc[j][2]);
      if constexpr (L::FULL8) {
        acc[j][3] = __ffma2_rn(ww, ex[0], acc[j][3]);
        acc[j][4] = __ffma2_rn(ww, ex[1], acc[j][4]);
      }
    }
  };

  // Words: offset q = (dy, dx), linear index l = dy SWS + dx: lower half
  // (l > 0) word l - 1 of the pixel, upper half word -l - 1 of the pixel at q.
  // So the word's place moves by `step` per offset: in the upper half back one
  // plane and on one column (at a row's end on to the next row's first), in
  // the lower half on one plane.  The words of the next run are in flight
  // while one is accumulated; word k is refilled as soon as it is used.
  const uint32_t plane = (uint32_t)G.rows * G.pitch;
  const Word* words = reinterpret_cast<const Word*>(vol + G.vol + G.pass[ps]);
  uint32_t off = lane_off + (uint32_t)(P.n_off / 2 - 1) * plane - (uint32_t)WSH * G.pitch - (uint32_t)WSH;
  uint32_t step = 1u - plane;
  const uint32_t row_step = (uint32_t)G.pitch - SWS;
  uint32_t buf[K];
  auto load = [&](int k) {
    buf[k] = __ldcg(words + off);
    off += step;
  };
#pragma unroll
  for (int k = 0; k < K; ++k) load(k);
  if (L::ROWRUNS == 1) off += row_step;
  const float4* v = reinterpret_cast<const float4*>(sm + L::OFF_CO) + warp * RO + lane;
  int rr = 1 % L::ROWRUNS;  // place of the next run in its window row
  for (int run = 0; run < L::RUNS; ++run) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float w[NP];
      if (k == K / 2 && run == L::MID) {
        // the centre: weight 1 (routines.cpp:151-157), read from memory: with
        // the constant the compiler folds w I^2 + A into one fused
        // multiply-add of I, rounded once instead of twice
        const float one = *reinterpret_cast<const float*>(sm + L::OFF_ONE);
#pragma unroll
        for (int j = 0; j < NP; ++j) w[j] = one;
      } else {
#pragma unroll
        for (int j = 0; j < NP; ++j) w[j] = weight(buf[k], j);
      }
      if (k == K / 2 && run + 1 == L::MID) {
        // the next run's centre has no word; its lower half starts at word 0
        off = lane_off;
        step = plane;
      } else if (run + 1 < L::RUNS) {
        load(k);
      }
      accumulate(w, v + k);
    }
    v += K;
    if (rr == 0) v += RO - SWS;  // this run was its row's last
    if (++rr == L::ROWRUNS) {
      rr = 0;
      // the run after the next starts a row
      if (run + 1 < L::MID) off += row_step;
    }
  }
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    float A[NA] = {sw[j], sww[j]};
#pragma unroll
    for (int a = 0; a < NA / 2 - 1; ++a) {
      A[2 + 2 * a] = acc[j][a].x;
      A[3 + 2 * a] = acc[j][a].y;
    }
    select_combo(P, pp.combo[j], A, 0, best);
  }
}

template <class L>
__global__ void __launch_bounds__(L::THREADS, 1)
    nlsar_mean_kernel(const __grid_constant__ FilterParams P, const SceneDesc* __restrict__ scenes,
                      const SplitSeg* __restrict__ segs, int nseg, const char* __restrict__ vol) {
  constexpr int WSH = L::WSH, RO = L::RO, NM = L::NM;
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  float4* sCo = reinterpret_cast<float4*>(sm + L::OFF_CO);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].tile_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const SplitSeg& G = segs[lo];
  const SceneDesc& S = scenes[G.scene];
  const int lt = (int)blockIdx.x - G.tile_begin;
  const int ty = lt / G.tiles_x, tx = lt - ty * G.tiles_x;
  const int vy0 = G.vy0 + ty * L::TH, vx0 = G.vx0 + tx * kTileW;

  // frame rows end at tiles of P.tile_h rows, so the last rows are clamped
  // (outputs that exist never use a clamped one)
  {
    const int Hp = S.tiles_y * P.tile_h + 2 * P.G;
    for (int r = warp; r < L::ROH; r += L::WARPS) {
      const size_t row = (size_t)min(vy0 - WSH + P.G + r, Hp - 1) * S.pitch + (vx0 - WSH + P.G);
#pragma unroll
      for (int q = 0; q < (RO + 31) / 32; ++q) {
        const int c = lane + 32 * q;
        if (c < RO) {
          sCo[r * RO + c] = S.cori[row + c];
          if constexpr (L::FULL8) sCo[L::PLANE + r * RO + c] = S.cori2[row + c];
        }
      }
    }
    if (tid == 0) *reinterpret_cast<float*>(sm + L::OFF_ONE) = 1.0f;
  }

  // pixels past the segment's last row and the last virtual column repeat it:
  // their words exist (columns are cut between tiles)
  const uint32_t lane_off = (uint32_t)(min(vy0 + warp, G.vy1 - 1) - G.row0) * G.pitch +
                            (uint32_t)(min(vx0 + lane, S.vW) - G.vx0) + WSH;

  Best<1, NM> best;
  best.e[0] = -1.0f;
  best.rank[0] = 0x7fffffff;
  best.combo[0] = -1;
  best.a[0] = 0.f;
  best.s0[0] = 1.f;
#pragma unroll
  for (int d = 0; d < NM; ++d) best.m[0][d] = 0.f;
  for (int ps = 0; ps < P.npass; ++ps) {
    // passes of one patch size come alone, others as three or two
    if constexpr (L::NPX == 1) {
      mean_pass<L, 1>(P, ps, vol, G, lane_off, best);
    } else if (P.pass[ps].np == 2) {
      mean_pass<L, 2>(P, ps, vol, G, lane_off, best);
    } else {
      mean_pass<L, 3>(P, ps, vol, G, lane_off, best);
    }
  }
  const int vy = vy0 + warp, vx = vx0 + lane;
  const int oy = (vy < S.H - 1) ? vy : (vy == S.vH ? S.H - 1 : -1);
  const int ox = (vx < S.W - 1) ? vx : (vx == S.vW ? S.W - 1 : -1);
  if (oy < 0 || ox < 0 || vy >= G.vy1) return;
  const int c = (warp + WSH) * RO + lane + WSH;
  float4 c2 = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (L::FULL8) c2 = sCo[L::PLANE + c];
  write_pixel<L::FULL8>(S, (size_t)oy * S.W + ox, sCo[c], c2, 0, best);
}

// Means as nlsar_kernels.cu sums them, any window: the offsets in pairs, the
// upper half's first and its mirror after it, the centre last.  One block: a
// 32 x TH tile, one pixel per thread, the window at run time.  Every setting
// measured gains over the kernel there, which computes every weight twice, a
// pixel's similarities, sums and weights behind three block barriers per few
// offsets: 400 x 450 with patches {3,5,7} and search 15 6.69 -> 0.88 ms, with
// {3,5} and search 21 9.56 -> 1.20 ms, search 3 0.32 -> 0.14 ms; 64 x 64 with
// one patch size and search 3 0.11 -> 0.07 ms.
constexpr int kPairs = 7;  // offset pairs whose words are in flight

__host__ __device__ constexpr int exact_tables(int npx) { return (npx + 1) / 2 * 65536; }
__host__ __device__ inline size_t exact_smem(int wsh, int th, bool full8, int npx) {
  return exact_tables(npx) + (size_t)(full8 ? 2 : 1) * (32 + 2 * wsh) * (th + 2 * wsh) * 16;
}

template <int TH, bool FULL8, int NPX>
struct ExactL {
  static constexpr int THREADS = 32 * TH;
  static constexpr int NA = FULL8 ? 12 : 8, NM = FULL8 ? 8 : 4;
};

template <int TH, bool FULL8, int NPX, int NP>
__device__ __forceinline__ void exact_pass(const FilterParams& P, int ps, const char* __restrict__ vol,
                                           const SplitSeg& G, uint32_t lane_off, int RO, int extra, float& best_e,
                                           float& best_a, float& best_s0, int& best_rank, int& best_combo,
                                           float* best_m) {
  using Word = typename WordOf<NP>::T;
  using L = ExactL<TH, FULL8, NPX>;
  constexpr int NA = L::NA;
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  const PassParams& pp = P.pass[ps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wsh = P.wsh;
  __syncthreads();  // the previous pass's tables are no longer read
  for (int i = tid; i < NP * 256 * 8; i += L::THREADS) {
    const int m = i >> 11, e = (i >> 3) & 255;
    const float w = e == kZeroCode ? 0.0f : P.wtab[pp.combo[m] * kMaxLut + e];
    *reinterpret_cast<float4*>(sm + (m >> 1) * 65536 + e * 256 + (m & 1) * 128 + (i & 7) * 16) =
        make_float4(w, w, w, w);
  }
  __syncthreads();
  float A[NP][NA];
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int a = 0; a < NA; ++a) A[j][a] = 0.0f;
  const uint32_t lane4 = 4u * lane;
  const float4* ctr = reinterpret_cast<const float4*>(sm + exact_tables(NPX)) + (warp + wsh) * RO + lane + wsh;
  auto accumulate = [&](uint32_t word, const float4* v) {
    const float4 c = v[0];
    float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (FULL8) e = v[extra];
    const float q0 = __fmul_rn(c.x, c.x), q1 = __fmul_rn(c.y, c.y);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const float w = *reinterpret_cast<const float*>(sm + (j >> 1) * 65536 + (j & 1) * 128 +
                                                      __byte_perm(word, lane4, 0x5504 | (j << 4)));
      A[j][0] = __fadd_rn(A[j][0], w);
      A[j][1] = __fmaf_rn(w, w, A[j][1]);
      A[j][2] = __fmaf_rn(w, c.x, A[j][2]);
      A[j][3] = __fmaf_rn(w, c.y, A[j][3]);
      A[j][4] = __fmaf_rn(w, q0, A[j][4]);
      A[j][5] = __fmaf_rn(w, q1, A[j][5]);
      A[j][6] = __fmaf_rn(w, c.z, A[j][6]);
      A[j][7] = __fmaf_rn(w, c.w, A[j][7]);
      if constexpr (FULL8) {
        A[j][8] = __fmaf_rn(w, e.x, A[j][8]);
        A[j][9] = __fmaf_rn(w, e.y, A[j][9]);
        A[j][10] = __fmaf_rn(w, e.z, A[j][10]);
        A[j][11] = __fmaf_rn(w, e.w, A[j][11]);
      }
    }
  };
  // pair i (offset o = (dy, dx) of the lower half, word i) from the last to
  // the first: the weight of -o is word i at x - o, of o word i at x
  const uint32_t plane = (uint32_t)G.rows * G.pitch;
  const Word* words = reinterpret_cast<const Word*>(vol + G.vol + G.pass[ps]);
  const int nhalf = P.n_off / 2;
  uint32_t up[kPairs], down[kPairs];
  int li = nhalf - 1, ldy = wsh, ldx = wsh;  // next pair to load
  auto load = [&](int k) {
    if (li >= 0) {
      const uint32_t off = lane_off + (uint32_t)li * plane;
      down[k] = __ldcg(words + off);
      up[k] = __ldcg(words + (off - (uint32_t)(ldy * G.pitch + ldx)));
      --li;
      if (--ldx < -wsh) ldx = wsh, --ldy;
    }
  };
#pragma unroll
  for (int k = 0; k < kPairs; ++k) load(k);
  int d = wsh * RO + wsh, dx = wsh;  // place of x + o after x
  for (int i = nhalf - 1; i >= 0; i -= kPairs) {
#pragma unroll
    for (int k = 0; k < kPairs; ++k) {
      if (i - k < 0) break;
      const uint32_t wu = up[k], wd = down[k];
      load(k);
      accumulate(wu, ctr - d);
      accumulate(wd, ctr + d);
      --d;
      if (--dx < -wsh) dx = wsh, d -= RO - 2 * wsh - 1;
    }
  }
  // centre weight 1, statistics, alpha, ENL', selection (nlsar_kernels.cu)
  const float4 c = ctr[0];
  float4 c2 = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (FULL8) c2 = ctr[extra];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const float s0 = A[j][0] + 1.0f, s1 = A[j][1] + 1.0f;
    const float s2 = A[j][2] + c.x, s3 = A[j][3] + c.y;
    // rounded as there, where the products are shared by the patch sizes
    const float s4 = __fadd_rn(A[j][4], __fmul_rn(c.x, c.x)), s5 = __fadd_rn(A[j][5], __fmul_rn(c.y, c.y));
    const float s6 = A[j][6] + c.z, s7 = A[j][7] + c.w;
    const float enl = s0 * s0 / s1;
    const float i0 = s2 / s0, i1 = s3 / s0;
    const float v0 = s4 / s0 - i0 * i0, v1 = s5 / s0 - i1 * i1;
    float alpha = 0.0f;
    alpha = fmaxf(alpha, fmaxf(0.0f, (v0 - i0 * i0) / v0));
    alpha = fmaxf(alpha, fmaxf(0.0f, (v1 - i1 * i1) / v1));
    if (P.alpha_zero) alpha = 0.0f;
    const float oma = 1.0f - alpha;
    const float enb = enl / (oma * oma + (alpha * alpha + 2.0f * alpha * (1.0f - alpha) / s0) * enl);
    const int combo = pp.combo[j];
    const int rank = P.combo[combo].rank;
    const bool take = P.select_mode == 0 || enb > best_e || (enb == best_e && rank < best_rank);
    const bool take_fb = !take && best_combo < 0 && combo == P.fallback_combo;
    if (take) {
      best_e = enb;
      best_rank = rank;
    }
    if (take || take_fb) {
      best_combo = combo;
      best_a = alpha;
      best_s0 = s0;
      best_m[0] = s2;
      best_m[1] = s3;
      best_m[2] = s6;
      best_m[3] = s7;
      if constexpr (FULL8) {
        best_m[4] = A[j][8] + c2.x;
        best_m[5] = A[j][9] + c2.y;
        best_m[6] = A[j][10] + c2.z;
        best_m[7] = A[j][11] + c2.w;
      }
    }
  }
}

template <int TH, bool FULL8, int NPX>
__global__ void __launch_bounds__(32 * TH, 1)
    nlsar_exact_mean_kernel(const __grid_constant__ FilterParams P, const SceneDesc* __restrict__ scenes,
                            const SplitSeg* __restrict__ segs, int nseg, const char* __restrict__ vol) {
  using L = ExactL<TH, FULL8, NPX>;
  extern __shared__ float4 smem4[];
  char* sm = reinterpret_cast<char*>(smem4);
  float4* sCo = reinterpret_cast<float4*>(sm + exact_tables(NPX));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wsh = P.wsh;
  const int RO = 32 + 2 * wsh, ROH = TH + 2 * wsh, extra = RO * ROH;
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].tile_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const SplitSeg& G = segs[lo];
  const SceneDesc& S = scenes[G.scene];
  const int lt = (int)blockIdx.x - G.tile_begin;
  const int ty = lt / G.tiles_x, tx = lt - ty * G.tiles_x;
  const int vy0 = G.vy0 + ty * TH, vx0 = G.vx0 + tx * kTileW;
  {
    const int Hp = S.tiles_y * P.tile_h + 2 * P.G;
    for (int r = warp; r < ROH; r += TH) {
      const size_t row = (size_t)min(vy0 - wsh + P.G + r, Hp - 1) * S.pitch + (vx0 - wsh + P.G);
      for (int c = lane; c < RO; c += 32) {
        sCo[r * RO + c] = S.cori[row + c];
        if constexpr (FULL8) sCo[extra + r * RO + c] = S.cori2[row + c];
      }
    }
  }
  // pixels past the segment's last row and the last virtual column repeat it:
  // their words exist (columns are cut between tiles)
  const uint32_t lane_off = (uint32_t)(min(vy0 + warp, G.vy1 - 1) - G.row0) * G.pitch +
                            (uint32_t)(min(vx0 + lane, S.vW) - G.vx0) + wsh;
  float best_e = -1.0f, alpha = 0.f, s0 = 1.f, m[L::NM];
  int best_rank = 0x7fffffff, combo = -1;
#pragma unroll
  for (int d = 0; d < L::NM; ++d) m[d] = 0.f;
  for (int ps = 0; ps < P.npass; ++ps) {
    auto pass = [&](auto np) {
      exact_pass<TH, FULL8, NPX, decltype(np)::value>(P, ps, vol, G, lane_off, RO, extra, best_e, alpha, s0, best_rank,
                                                      combo, m);
    };
    if constexpr (NPX == 1) {
      pass(std::integral_constant<int, 1>{});
    } else if (P.pass[ps].np == 2) {
      pass(std::integral_constant<int, 2>{});
    } else {
      pass(std::integral_constant<int, 3>{});
    }
  }
  const int vy = vy0 + warp, vx = vx0 + lane;
  const int oy = (vy < S.H - 1) ? vy : (vy == S.vH ? S.H - 1 : -1);
  const int ox = (vx < S.W - 1) ? vx : (vx == S.vW ? S.W - 1 : -1);
  if (oy < 0 || ox < 0 || vy >= G.vy1) return;
  const float4 c = sCo[(warp + wsh) * RO + lane + wsh];
  const float oma = 1.0f - alpha;
  const float c00 = oma * m[0] / s0 + alpha * c.x;
  const float c11 = oma * m[1] / s0 + alpha * c.y;
  const float cre = oma * m[2] / s0 + alpha * c.z;
  const float cim = oma * m[3] / s0 + alpha * c.w;
  const size_t o = (size_t)oy * S.W + ox;
  if constexpr (FULL8) {
    const float4 c2 = sCo[extra + (warp + wsh) * RO + lane + wsh];
    const size_t n = (size_t)S.H * S.W;
    S.cov_out[o] = c00;
    S.cov_out[n + o] = oma * m[4] / s0 + alpha * c2.x;
    S.cov_out[2 * n + o] = cre;
    S.cov_out[3 * n + o] = cim;
    S.cov_out[4 * n + o] = oma * m[5] / s0 + alpha * c2.y;
    S.cov_out[5 * n + o] = oma * m[6] / s0 + alpha * c2.z;
    S.cov_out[6 * n + o] = c11;
    S.cov_out[7 * n + o] = oma * m[7] / s0 + alpha * c2.w;
  } else {
    const float am = sqrtf(c00), as = sqrtf(c11);
    const float r = 0.5f * (am + as);
    S.ref[o] = r * r;
    S.phase[o] = atan2f(cim, cre);
    S.coh[o] = sqrtf(cim * cim + cre * cre) / (am * as);
  }
  if (S.sel_out) S.sel_out[o] = combo;
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------

// pass shapes with an index kernel: 0 {1,2,3}, 1 {4,5}, 2..6 the single
// halves 1..5, 7 {1,2}; -1 none
int pass_shape(const PassParams& p) {
  if (p.np == 3 && p.ph[0] == 1 && p.ph[1] == 2 && p.ph[2] == 3) return 0;
  if (p.np == 2 && p.ph[0] == 4 && p.ph[1] == 5) return 1;
  if (p.np == 1 && p.ph[0] >= 1 && p.ph[0] <= 5) return 1 + p.ph[0];
  if (p.np == 2 && p.ph[0] == 1 && p.ph[1] == 2) return 7;
  return -1;
}
int shape_phm(int shape) { return shape == 0 ? 3 : (shape == 1 ? 5 : (shape == 7 ? 2 : shape - 1)); }
int shape_vc(int shape) { return 128 - 8 * ((shape_phm(shape) + 3) / 4); }

template <int PH0, int PH1, int PH2, bool EXACT>
cudaError_t launch_index_t(const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                           const PassList& passes, int slot, char* vol, dim3 grid, size_t smem,
                           cudaStream_t st) {
  static size_t allowed[kMaxDevices];
  const cudaError_t e = allow_dynamic_smem((const void*)nlsar_index_kernel<PH0, PH1, PH2, EXACT>, smem, allowed);
  if (e != cudaSuccess) return e;
  nlsar_index_kernel<PH0, PH1, PH2, EXACT><<<grid, kIdxThreads, smem, st>>>(F, scenes, segs, nseg, passes, slot, vol);
  return cudaGetLastError();
}

template <int TH, bool FULL8, int NPX>
cudaError_t launch_mean_t(const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                          const char* vol, int tiles, cudaStream_t st) {
  using L = MeanL<10, TH, FULL8, NPX>;
  static size_t allowed[kMaxDevices];
  const cudaError_t e = allow_dynamic_smem((const void*)nlsar_mean_kernel<L>, L::BYTES, allowed);
  if (e != cudaSuccess) return e;
  nlsar_mean_kernel<L><<<tiles, L::THREADS, L::BYTES, st>>>(F, scenes, segs, nseg, vol);
  return cudaGetLastError();
}

// Rows of the tallest mean tile: 32, with 8-plane input 16 (its accumulators
// want more registers; 24 rows measured 4.39 ms against 4.17 at 1100 x 1203)
constexpr int tall_tile(bool full8) { return full8 ? 16 : 32; }

template <bool FULL8, int NPX>
cudaError_t launch_mean_th(int th, const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                           const char* vol, int tiles, cudaStream_t st) {
  if (th == 8) return launch_mean_t<8, FULL8, NPX>(F, scenes, segs, nseg, vol, tiles, st);
  if (th == 16) return launch_mean_t<16, FULL8, NPX>(F, scenes, segs, nseg, vol, tiles, st);
  return launch_mean_t<tall_tile(FULL8), FULL8, NPX>(F, scenes, segs, nseg, vol, tiles, st);
}

template <int TH, bool FULL8, int NPX>
cudaError_t launch_exact_t(const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                           const char* vol, int tiles, cudaStream_t st) {
  const size_t smem = exact_smem(F.wsh, TH, FULL8, NPX);
  static size_t allowed[kMaxDevices];
  const cudaError_t e =
      allow_dynamic_smem((const void*)nlsar_exact_mean_kernel<TH, FULL8, NPX>, kSplitSmem, allowed);
  if (e != cudaSuccess) return e;
  nlsar_exact_mean_kernel<TH, FULL8, NPX><<<tiles, 32 * TH, smem, st>>>(F, scenes, segs, nseg, vol);
  return cudaGetLastError();
}

template <bool FULL8, int NPX>
cudaError_t launch_exact_th(int th, const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                            const char* vol, int tiles, cudaStream_t st) {
  if (th == 8) return launch_exact_t<8, FULL8, NPX>(F, scenes, segs, nseg, vol, tiles, st);
  if (th == 16) return launch_exact_t<16, FULL8, NPX>(F, scenes, segs, nseg, vol, tiles, st);
  return launch_exact_t<tall_tile(FULL8), FULL8, NPX>(F, scenes, segs, nseg, vol, tiles, st);
}

bool single_patches(const FilterParams& F) {
  for (int i = 0; i < F.npass; ++i)
    if (F.pass[i].np > 1) return false;
  return true;
}

size_t word_bytes(int np) { return np == 3 ? 4 : np; }

int div_up(int a, int b) { return (a + b - 1) / b; }

}  // namespace

bool split_supported(const Plan& pl) {
  const FilterParams& F = pl.P;
  if (F.prec != 0 || F.withhold_staging || !split_tables_ok(pl)) return false;
  if (pl.fast) return true;
  // settings of the kernel in nlsar_kernels.cu: passes that the index kernel
  // has (their sizes in any scale), and a window whose staged planes fit
  if (pl.generic_only || F.npass < 1) return false;
  int shapes = 0, seen[kMaxPasses];
  for (int i = 0; i < F.npass; ++i) {
    const int s = pass_shape(F.pass[i]);
    if (s < 0) return false;
    int k = 0;
    while (k < shapes && seen[k] != s) ++k;
    if (k == shapes) seen[shapes++] = s;
    if (idx_smem(F.wsh, shape_phm(s), 8) > kSplitSmem) return false;
  }
  const int npx = single_patches(F) ? 1 : 3;
  if (npx == 3)
    for (int i = 0; i < F.npass; ++i)
      if (F.pass[i].np == 1) return false;  // the mean kernels take passes of one size alone
  return shapes <= kSplitShapes && F.wsh >= 1 && idx_left(F.wsh) + 128 + F.wsh <= 32 * kIdxLoads &&
         exact_smem(F.wsh, tall_tile(pl.full8), pl.full8, npx) <= kSplitSmem;
}

bool split_tables_ok(const Plan& pl) {
  const FilterParams& F = pl.P;
  for (int i = 0; i < F.npass; ++i)
    for (int j = 0; j < F.pass[i].np; ++j) {
      const int c = F.pass[i].combo[j];
      const float* w = pl.wtab.data() + (size_t)c * kMaxLut;
      if (F.combo[c].lm1 > 254.0f && std::memcmp(w + 254, w + 255, sizeof(float)) != 0) return false;
    }
  return true;
}

size_t split_budget() {
  if (const char* v = std::getenv("DESPECKCL_B200_VOLUME_MIB")) {
    char* end = nullptr;
    const unsigned long long mib = std::strtoull(v, &end, 10);
    if (end != v && mib < (kSplitBudgetBytes >> 20)) return (size_t)mib << 20;
  }
  return kSplitBudgetBytes;
}

// Cuts the jobs (row ranges of scenes) into segments of at most `budget`
// bytes of volume, groups the segments into chunks of at most that size, and
// chooses every chunk's block rows and offset groups.  Segments are runs of
// whole rows where a row of the tallest tiles fits; else such rows are cut in
// columns too.  False where one tile with its window does not fit.
bool split_layout(const Plan& pl, const std::vector<SceneGeom>& geo, const std::vector<SplitJob>& jobs,
                  size_t budget, int sms, SplitLayout& out) {
  const FilterParams& F = pl.P;
  const int big = tall_tile(pl.full8);  // segments hold whole tiles
  const int nhalf = F.n_off / 2;
  out.segs.clear();
  out.chunks.clear();
  out.vol_bytes = 0;
  // the call's pass shapes, in order of first use
  out.nshape = 0;
  for (int i = 0; i < F.npass; ++i) {
    const int s = pass_shape(F.pass[i]);
    int k = 0;
    while (k < out.nshape && out.shape[k] != s) ++k;
    if (k == out.nshape) {
      out.shape[out.nshape] = s;
      out.passes[out.nshape++].n = 0;
    }
    out.passes[k].id[out.passes[k].n++] = i;
  }
  auto pitch_of = [&](int cols) { return (cols + 2 * F.wsh + 3) / 4 * 4; };
  // bytes of a segment's volume, and whether it may be one: the mean kernels'
  // word offsets within a pass are 32-bit
  auto volume = [&](int rows, int cols, size_t* pass) {
    size_t bytes = 0;
    for (int p = 0; p < F.npass; ++p) {
      if (pass) pass[p] = bytes;
      bytes += ((size_t)nhalf * (rows + F.wsh) * pitch_of(cols) * word_bytes(F.pass[p].np) + 255) / 256 * 256;
    }
    return bytes;
  };
  auto fits = [&](int rows, int cols) {
    return volume(rows, cols, nullptr) <= budget && (size_t)nhalf * (rows + F.wsh) * pitch_of(cols) <= 0x3fffffff;
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
  size_t used = 0;
  auto close_chunk = [&] {
    if (!out.chunks.empty()) out.chunks.back().seg1 = (int)out.segs.size();
    used = 0;
  };
  for (const SplitJob& j : jobs) {
    const SceneGeom& g = geo[j.scene];
    const int row1 = std::min(j.row1, g.vH + 1), width = g.vW + 1;
    if (j.row0 >= row1) continue;
    const int n = row1 - j.row0;
    int wide = width, rows = largest(div_up(n, big) * big, big, [&](int r) { return fits(std::min(r, n), width); });
    if (rows == 0) {
      rows = big;
      wide = largest(div_up(width, kTileW) * kTileW, kTileW, [&](int c) { return fits(std::min(big, n), c); });
      if (wide == 0) return false;
      wide = div_up(div_up(width, div_up(width, wide)), kTileW) * kTileW;
    }
    const int step = div_up(div_up(n, div_up(n, rows)), big) * big;
    for (int y = j.row0; y < row1; y += step)
      for (int x = 0; x < width; x += wide) {
        SplitSeg s{};
        s.scene = j.scene;
        s.vy0 = y;
        s.vy1 = std::min(y + step, row1);
        const int cols = std::min(wide, width - x);
        s.vx0 = x;
        s.row0 = y - F.wsh;
        s.rows = s.vy1 - s.row0;
        s.pitch = pitch_of(cols);
        s.tiles_x = div_up(cols, kTileW);
        const size_t bytes = volume(s.vy1 - s.vy0, cols, s.pass);
        if (out.chunks.empty() || (used && used + bytes > budget)) {
          close_chunk();
          out.chunks.push_back(SplitChunk{});
          out.chunks.back().seg0 = (int)out.segs.size();
        }
        s.vol = used;
        used += bytes;
        out.vol_bytes = std::max(out.vol_bytes, used);
        out.segs.push_back(s);
      }
  }
  close_chunk();
  for (SplitChunk& c : out.chunks) {
    // Rows of the mean tiles: waves of blocks (one per SM) times a block's
    // time, measured at 1024^2: 182, 94 and 59 us for 32, 16 and 8 rows (few
    // warps leave latency uncovered), in proportion for other patch sets
    double best_t = 0.0;
    for (int th : {big, 16, 8}) {
      int tiles = 0;
      for (int i = c.seg0; i < c.seg1; ++i)
        tiles += out.segs[i].tiles_x * div_up(out.segs[i].vy1 - out.segs[i].vy0, th);
      const double t = (double)div_up(tiles, sms) * (th > 16 ? 182.0 : (th > 8 ? 94.0 : 59.0));
      if (best_t == 0.0 || t < 0.98 * best_t) {
        best_t = t;
        c.th = th;
        c.tiles = tiles;
      }
    }
    int tiles = 0;
    for (int i = c.seg0; i < c.seg1; ++i) {
      SplitSeg& s = out.segs[i];
      s.tile_begin = tiles;
      tiles += s.tiles_x * div_up(s.vy1 - s.vy0, c.th);
    }
    for (int k = 0; k < out.nshape; ++k) {
      // Block rows R and offset groups Z: the time of a chunk is its waves of
      // blocks (one per SM) times a block's time, staging (about 0.1 us per
      // staged row) plus its rounds of 16 offsets (about 0.5 us per row that
      // a round walks, patch halo included).  Large chunks take the tallest
      // blocks; scenes of few blocks are spread over all SMs.
      const int phm = shape_phm(out.shape[k]), vc = shape_vc(out.shape[k]);
      int rmax = 1;
      while (idx_smem(F.wsh, phm, rmax + 1) <= kSplitSmem) ++rmax;
      double best = 0.0;
      int best_r = rmax, best_z = 1;
      for (int r = rmax; r >= std::min(rmax, 8); r -= (r > 16 ? 2 : 1)) {
        long long blocks = 0;
        int tall = 0;
        for (int i = c.seg0; i < c.seg1; ++i) {
          const SplitSeg& s = out.segs[i];
          const int by = div_up(s.rows, r);
          tall = std::max(tall, div_up(s.rows, by));
          blocks += (long long)div_up(s.pitch, vc) * by;
        }
        blocks *= out.passes[k].n;
        for (int z = 1; z <= div_up(nhalf, kIdxWarps); ++z) {
          const int rounds = div_up(nhalf, kIdxWarps * z);
          const double t = (double)((blocks * z + sms - 1) / sms) *
                           (2.0 + 0.1 * (tall + 2 * phm + F.wsh) + 0.5 * rounds * (tall + 2 * phm));
          if (best == 0.0 || t < best * 0.999) {
            best = t;
            best_r = r;
            best_z = z;
          }
        }
      }
      int blocks = 0, rows = 1;
      for (int i = c.seg0; i < c.seg1; ++i) {
        SplitSeg& s = out.segs[i];
        const int by = div_up(s.rows, best_r);
        s.idx_R[k] = div_up(s.rows, by);
        s.idx_bx[k] = div_up(s.pitch, vc);
        s.idx_begin[k] = blocks;
        rows = std::max(rows, s.idx_R[k]);
        blocks += s.idx_bx[k] * div_up(s.rows, s.idx_R[k]);
      }
      c.idx_blocks[k] = blocks;
      c.idx_z[k] = best_z;
      c.idx_smem[k] = idx_smem(F.wsh, phm, rows);
    }
  }
  return true;
}

int split_launches(const SplitLayout& lay) { return (int)lay.chunks.size() * (lay.nshape + 1); }

cudaError_t launch_split(const Plan& pl, const FilterParams& F, const SplitLayout& lay, int chunk,
                         const SceneDesc* d_scenes, const SplitSeg* d_segs, char* vol, cudaStream_t st) {
  const SplitChunk& c = lay.chunks[chunk];
  const SplitSeg* segs = d_segs + c.seg0;
  const int nseg = c.seg1 - c.seg0;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < lay.nshape && e == cudaSuccess; ++k) {
    const dim3 grid(c.idx_blocks[k], c.idx_z[k], lay.passes[k].n);
    auto go = [&](auto launch) {
      return launch(F, d_scenes, segs, nseg, lay.passes[k], k, vol, grid, c.idx_smem[k], st);
    };
    auto index = [&](auto exact) {
      constexpr bool EXACT = decltype(exact)::value;
      switch (lay.shape[k]) {
        case 0: return go(launch_index_t<1, 2, 3, EXACT>);
        case 1: return go(launch_index_t<4, 5, -1, EXACT>);
        case 2: return go(launch_index_t<1, -1, -1, EXACT>);
        case 3: return go(launch_index_t<2, -1, -1, EXACT>);
        case 4: return go(launch_index_t<3, -1, -1, EXACT>);
        case 5: return go(launch_index_t<4, -1, -1, EXACT>);
        case 6: return go(launch_index_t<5, -1, -1, EXACT>);
        case 7: return EXACT ? go(launch_index_t<1, 2, -1, true>) : cudaErrorInvalidValue;
        default: return cudaErrorInvalidValue;
      }
    };
    e = pl.fast ? index(std::false_type{}) : index(std::true_type{});
  }
  if (e != cudaSuccess) return e;
  const bool single = single_patches(F);
  auto mean = [&](auto full8, auto npx) {
    constexpr bool FULL8 = decltype(full8)::value;
    constexpr int NPX = decltype(npx)::value;
    return pl.fast ? launch_mean_th<FULL8, NPX>(c.th, F, d_scenes, segs, nseg, vol, c.tiles, st)
                   : launch_exact_th<FULL8, NPX>(c.th, F, d_scenes, segs, nseg, vol, c.tiles, st);
  };
  using one = std::integral_constant<int, 1>;
  using three = std::integral_constant<int, 3>;
  if (pl.full8) return single ? mean(std::true_type{}, one{}) : mean(std::true_type{}, three{});
  return single ? mean(std::false_type{}, one{}) : mean(std::false_type{}, three{});
}

}  // namespace dcl

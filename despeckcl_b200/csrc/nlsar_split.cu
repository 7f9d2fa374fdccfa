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
//      the index of the composite weight (compute_weights.cl:40-51); up to
//      three patch sizes of a pass share one 32-bit word per (offset, pixel).
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
// The volume of one pass is (sws^2 - 1) / 2 words per pixel (880 B at search
// 21), so a scene is filtered in segments of rows whose volume fits a budget
// (kSplitBudgetBytes), index kernel and mean kernel in turn.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "dcl_internal.h"
#include "nlsar_math.cuh"
#include "nlsar_split.h"

namespace dcl {

namespace {

// A weight's field in a word: 9 bits, the table entry or kZeroField.  Field j
// sits at bits 6 + 9 j (the third wraps around), so that a masked word (the
// second and third field after a shift or rotation) is the byte offset of the
// entry in a table with 16 interleaved copies.
constexpr int kZeroField = 256;
constexpr int kLutCopies = 16;
constexpr int kOneField = 257;  // the centre's weight
constexpr int kLutWords = (kOneField + 1) * kLutCopies;  // one table
constexpr uint32_t kFieldMask = 0x1FFu << 6;

constexpr int kIdxWarps = 16;
constexpr int kIdxThreads = 32 * kIdxWarps;

template <int PHM>
struct IdxL {
  // lanes own four adjacent columns; HL lanes at each end of a warp only
  // supply the patch halo
  static constexpr int HL = (PHM + 3) / 4;
  static constexpr int VC = 128 - 8 * HL;  // columns a warp produces
};

__host__ __device__ inline int idx_left(int wsh) { return (wsh + 3) / 4 * 4; }  // staged columns left of lane 0
// float4 slots of a staged row: five per four pixels (see the kernel)
__host__ __device__ inline int idx_row_slots(int wsh) { return 5 * ((idx_left(wsh) + 128 + wsh + 3) / 4); }
__host__ __device__ inline size_t idx_smem(int wsh, int phm, int R) {
  return (size_t)(R + 2 * phm + wsh) * idx_row_slots(wsh) * 20;
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
// A warp walks down the rows for one offset.  Per row a lane evaluates four
// similarities, gets the patch halo from its neighbour lanes by shuffles,
// forms the horizontal sums in the nested-ring order of the fused kernel, and
// keeps, per patch size 2 ph + 1, the 2 ph partial vertical sums in flight
// (the sum of the last k rows, top down), so a vertical sum costs 2 ph adds,
// two columns per packed add, and no loads.  A smaller patch is complete
// PHM - ph rows before the largest, so its field waits in `pend`.
template <int PH0, int PH1, int PH2>
__global__ void __launch_bounds__(kIdxThreads, 1)
    nlsar_index_kernel(const __grid_constant__ FilterParams P, const SceneDesc* __restrict__ scenes,
                       const SplitSeg* __restrict__ segs, int nseg, const __grid_constant__ PassList passes,
                       int shape, uint32_t* __restrict__ vol) {
  constexpr int NP = np_of<PH0, PH1, PH2>();
  constexpr int PHM = cmax(PH0, cmax(PH1, PH2));
  constexpr int HL = IdxL<PHM>::HL, VC = IdxL<PHM>::VC;
  constexpr int ND = PHM - PH0;  // rows the first patch's field waits
  static_assert(PH0 >= 1 && 4 * HL >= PHM, "pass shape");
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
    // c is virtual column c - wsh.  Coordinates are clamped to the frame: the
    // pixels a used weight needs are inside it.
    const int Hp = D.tiles_y * P.tile_h + 2 * P.G, Wp = D.tiles_x * kTileW + 2 * P.G;
    const int fx0 = VC * bx - 4 * HL - wsh - left + P.G, fy0 = S.row0 + r0 - PHM + P.G;
    const int ncol = left + 128 + wsh;
    const float4* cs = D.cs[pp.scale_slot];
    constexpr int U = 6;  // 32 U >= ncol for search windows up to 41
    for (int r = warp; r < nrow; r += kIdxWarps) {
      const float4* row = cs + (size_t)min(max(fy0 + r, 0), Hp - 1) * D.pitch;
      float4 v[U];
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (lane + 32 * k < ncol) v[k] = row[min(max(fx0 + lane + 32 * k, 0), Wp - 1)];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int p = lane + 32 * k;
        if (p < ncol) {
          const int slot = r * SP + p + (p >> 2);
          const float t = pixel_term<kPrecRatio>(v[k]);
          sC[slot] = v[k];
          sL[slot] = t;
          reinterpret_cast<float*>(sC + r * SP + 5 * (p >> 2) + 4)[p & 3] = t;
        }
      }
    }
  }
  // patch sums are in log2 units: the lookup scales by ln 2 (nlsar_fast.cu)
  float inv_span[NP], nbias[NP], lm1[NP], dmax[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const ComboParams& cp = P.combo[pp.combo[j]];
    inv_span[j] = 1.0f / cp.span;
    nbias[j] = -cp.dmin * inv_span[j];
    lm1[j] = cp.lm1;
    dmax[j] = cp.dmax;
    inv_span[j] *= 0.69314718f;
    dmax[j] *= 1.44269504f;
  }
  __syncthreads();

  const int nhalf = P.n_off / 2;
  const int c = VC * bx + 4 * (lane - HL);  // this lane's first volume column
  const bool writes = lane >= HL && lane < 32 - HL && c < S.pitch;
  const size_t plane = (size_t)S.rows * S.pitch;
  uint32_t* out0 = vol + S.vol + (size_t)ps * nhalf * plane + (size_t)r0 * S.pitch + c;

  for (int u = (int)blockIdx.y * kIdxWarps + warp; u < nhalf; u += kIdxWarps * (int)gridDim.y) {
    // lower half window, row-major: (0, 1) .. (0, wsh), (1, -wsh) ..
    const int v = u + wsh + 1;
    const int dy = v / sws, dx = v - dy * sws - wsh;
    const float4* ctr = sC + 5 * (lane + (left >> 2));
    int ns[4];  // slots of the four neighbours
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int t = left + dx + j;
      ns[j] = dy * SP + 5 * (lane + (t >> 2)) + (t & 3);
    }
    // partial vertical sums: vs[j][k]: last k + 1 rows of patch j, columns in pairs
    float2 vs[NP][2 * PHM][2];
    uint32_t pend[ND > 0 ? ND : 1][4];
#pragma unroll
    for (int j = 0; j < NP; ++j)
#pragma unroll
      for (int k = 0; k < 2 * PHM; ++k)
#pragma unroll
        for (int q = 0; q < 2; ++q) vs[j][k][q] = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < ND; ++k)
#pragma unroll
      for (int o = 0; o < 4; ++o) pend[k][o] = 0;
    uint32_t* out = out0 + (size_t)u * plane;
    for (int i = 0; i < R + 2 * PHM; ++i) {
      // ---- similarities of the lane's four columns
      float s[4 + 2 * PHM];
      {
        const float4 la = ctr[4];
        const float la4[4] = {la.x, la.y, la.z, la.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) s[PHM + j] = glr_sim<kPrecRatio>(ctr[j], la4[j], sC[ns[j]], sL[ns[j]], 0.0f);
      }
      ctr += SP;
#pragma unroll
      for (int j = 0; j < 4; ++j) ns[j] += SP;
#pragma unroll
      for (int k = 1; k <= PHM; ++k) {
        s[PHM - k] = __shfl_up_sync(0xffffffffu, s[PHM + 3 - (k - 1) % 4], (k + 3) / 4);
        s[PHM + 3 + k] = __shfl_down_sync(0xffffffffu, s[PHM + (k - 1) % 4], (k + 3) / 4);
      }
      // ---- horizontal sums (nested rings)
      float hs[NP][4];
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        float ring = s[o + PHM];
#pragma unroll
        for (int b = 1; b <= PHM; ++b) {
          ring += s[o + PHM - b] + s[o + PHM + b];
#pragma unroll
          for (int j = 0; j < NP; ++j)
            if (ph_of<PH0, PH1, PH2>(j) == b) hs[j][o] = ring;
        }
      }
      // ---- vertical sums, the weight's table index
      uint32_t field[NP][4];
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const int n = 2 * ph_of<PH0, PH1, PH2>(j);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 h = make_float2(hs[j][2 * q], hs[j][2 * q + 1]);
          const float2 d2 = __fadd2_rn(vs[j][n - 1][q], h);
#pragma unroll
          for (int k = n - 1; k > 0; --k) vs[j][k][q] = __fadd2_rn(vs[j][k - 1][q], h);
          vs[j][0][q] = h;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float d = e ? d2.y : d2.x;
            // saturating FMA (clamps, NaN to 0), round-toward-zero add of
            // 2^23: the low mantissa bits are the index; d > dmax: weight 0
            const float uu = __saturatef(fmaf(d, inv_span[j], nbias[j]));
            const float t = __fmaf_rz(uu, lm1[j], 8388608.0f);
            field[j][2 * q + e] = d > dmax[j] ? 0x4B000000u + kZeroField : __float_as_uint(t);
          }
        }
      }
      // ---- the words of row i - 2 PHM; the exponent bits of field 0 are
      // taken out, those of the others are shifted out
      uint32_t w[4];
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        auto part = [&](int wait) {
          uint32_t f = 0;
#pragma unroll
          for (int j = 0; j < NP; ++j)
            if (PHM - ph_of<PH0, PH1, PH2>(j) == wait)
              f += j == 0 ? field[0][o] - 0x4B000000u : field[j][o] << (9 * j);
          return f;
        };
        w[o] = (ND > 0 ? pend[0][o] : 0u) + part(0);
#pragma unroll
        for (int k = 0; k < ND; ++k) pend[k][o] = (k + 1 < ND ? pend[k + 1][o] : 0u) + part(k + 1);
        w[o] = __funnelshift_l(w[o], w[o], 6);
      }
      if (i >= 2 * PHM) {
        if (writes) *reinterpret_cast<uint4*>(out) = make_uint4(w[0], w[1], w[2], w[3]);
        out += S.pitch;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// mean kernel
// ---------------------------------------------------------------------------

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Tile rows, threads and shared memory: 32 x TH outputs, two vertically
// adjacent pixels per thread (their accumulators packed in pairs).  InSAR
// input: 16 rows, 8 warps, two blocks per SM; 8-plane input: 24 rows, 12
// warps, one block per SM (12 accumulators per pixel and patch size).
template <bool FULL8>
struct MeanL {
  static constexpr int TH = FULL8 ? kSplitTileH8 : kSplitTileH, PX = 2;
  static constexpr int WARPS = TH / PX, THREADS = 32 * WARPS;
  static constexpr int BLOCKS = FULL8 ? 1 : 2;
  static constexpr int NA = FULL8 ? 12 : 8, NM = FULL8 ? 8 : 4;
};

__host__ __device__ inline int mean_region(int wsh, int th) { return (32 + 2 * wsh) * (th + 2 * wsh); }
// float4 planes, then the weight tables, then one {volume, tile} offset pair
// per search-window position
__host__ __device__ inline size_t mean_smem(int wsh, int np, bool full8, int n_off) {
  const int th = full8 ? kSplitTileH8 : kSplitTileH;
  return (size_t)mean_region(wsh, th) * 16 * (full8 ? 2 : 1) + (size_t)np * kLutWords * 4 + (size_t)n_off * 8;
}

// One pass of NP patch sizes over the window: `words` points at the thread's
// first pixel in the pass's volume.
template <int NP, bool FULL8>
__device__ __forceinline__ void mean_pass(const FilterParams& P, const PassParams& pp, const uint32_t* words,
                                          int wpitch, const float4* sCo, const float4* sCo2, float* sLut,
                                          const int2* sOff, int RO, int ci,
                                          Best<MeanL<FULL8>::PX, MeanL<FULL8>::NM>& best) {
  using L = MeanL<FULL8>;
  constexpr int PX = L::PX, NA = L::NA;
  const int tid = threadIdx.x, lane = tid & 31;
  __syncthreads();  // the previous pass's tables are no longer read
  for (int i = tid; i < NP * kLutWords; i += L::THREADS) {
    const int j = i / kLutWords;
    const int e = (i - j * kLutWords) / kLutCopies;
    sLut[i] = e < kMaxLut ? P.wtab[pp.combo[j] * kMaxLut + e] : (e == kOneField ? 1.0f : 0.0f);
  }
  __syncthreads();
  float2 acc[NP][NA];  // .x: the upper pixel, .y: the lower one
#pragma unroll
  for (int j = 0; j < NP; ++j)
#pragma unroll
    for (int a = 0; a < NA; ++a) acc[j][a] = make_float2(0.f, 0.f);
  const uint32_t copy = 4u * (lane & (kLutCopies - 1));
  const char* lut = reinterpret_cast<const char*>(sLut);

  // two pixels per packed (f32x2) operation; each component is rounded like
  // the scalar add / multiply / fma
  auto accumulate = [&](const float2 (&ww)[NP], int oa) {
    const float4 va = sCo[oa], vb = sCo[oa + RO];
    const float2 vx = make_float2(va.x, vb.x), vy = make_float2(va.y, vb.y);
    const float2 vz = make_float2(va.z, vb.z), vw = make_float2(va.w, vb.w);
    const float2 x2 = __fmul2_rn(vx, vx), y2 = __fmul2_rn(vy, vy);
    float2 ex[4];
    if (FULL8) {
      const float4 ea = sCo2[oa], eb = sCo2[oa + RO];
      ex[0] = make_float2(ea.x, eb.x);
      ex[1] = make_float2(ea.y, eb.y);
      ex[2] = make_float2(ea.z, eb.z);
      ex[3] = make_float2(ea.w, eb.w);
    }
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      float2* A = acc[j];
      A[0] = __fadd2_rn(A[0], ww[j]);
      A[1] = __ffma2_rn(ww[j], ww[j], A[1]);
      A[2] = __ffma2_rn(ww[j], vx, A[2]);
      A[3] = __ffma2_rn(ww[j], vy, A[3]);
      A[4] = __ffma2_rn(ww[j], x2, A[4]);
      A[5] = __ffma2_rn(ww[j], y2, A[5]);
      A[6] = __ffma2_rn(ww[j], vz, A[6]);
      A[7] = __ffma2_rn(ww[j], vw, A[7]);
      if (FULL8) {
#pragma unroll
        for (int e = 0; e < 4; ++e) A[(8 + e) % NA] = __ffma2_rn(ww[j], ex[e], A[(8 + e) % NA]);
      }
    }
  };
  auto weight = [&](uint32_t w, int j) {
    const uint32_t f = j == 0 ? w : (j == 1 ? w >> 9 : __funnelshift_r(w, w, 18));
    return *reinterpret_cast<const float*>(lut + j * kLutWords * 4 + ((f & kFieldMask) | copy));
  };

  // words of the next D offsets in flight while D are accumulated (their
  // latency is that of HBM; n_off is a multiple of 8)
  constexpr int D = 4;
  const int n = P.n_off;
  uint32_t nxt[D][PX];
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const uint32_t* p = words + sOff[k].x;
    nxt[k][0] = __ldcg(p);
    nxt[k][1] = __ldcg(p + wpitch);
  }
  for (int t = 0; t < n; t += D) {
    uint32_t cur[D][PX];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      cur[k][0] = nxt[k][0];
      cur[k][1] = nxt[k][1];
    }
    if (t + D < n) {
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const uint32_t* p = words + sOff[t + D + k].x;
        nxt[k][0] = __ldcg(p);
        nxt[k][1] = __ldcg(p + wpitch);
      }
    }
    if (2 * t == n) {  // the centre, between the two halves (routines.cpp:151-157)
      // weight 1 from the table: with the constant the compiler folds w I^2 + A
      // into one fused multiply-add of I, rounded once instead of twice
      float2 ww[NP];
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const float one = sLut[j * kLutWords + kOneField * kLutCopies];
        ww[j] = make_float2(one, one);
      }
      accumulate(ww, ci);
    }
#pragma unroll
    for (int k = 0; k < D; ++k) {
      float2 ww[NP];
#pragma unroll
      for (int j = 0; j < NP; ++j) ww[j] = make_float2(weight(cur[k][0], j), weight(cur[k][1], j));
      accumulate(ww, ci + sOff[t + k].y);
    }
  }
#pragma unroll
  for (int i = 0; i < PX; ++i)
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      float A[NA];
#pragma unroll
      for (int a = 0; a < NA; ++a) A[a] = (i & 1) ? acc[j][a].y : acc[j][a].x;
      select_combo(P, pp.combo[j], A, i, best);
    }
}

// One block: one 32 x TH tile of a segment, all passes.
template <int NPX, bool FULL8>
__global__ void __launch_bounds__(MeanL<FULL8>::THREADS, MeanL<FULL8>::BLOCKS)
    nlsar_mean_kernel(const __grid_constant__ FilterParams P, const SceneDesc* __restrict__ scenes,
                      const SplitSeg* __restrict__ segs, int nseg, const uint32_t* __restrict__ vol) {
  using L = MeanL<FULL8>;
  constexpr int PX = L::PX, NM = L::NM;
  extern __shared__ float4 smem4[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].tile_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const SplitSeg G = segs[lo];
  const SceneDesc& S = scenes[G.scene];
  const int lt = (int)blockIdx.x - G.tile_begin;
  const int ty = lt / G.tiles_x, tx = lt - ty * G.tiles_x;
  const int vy0 = G.vy0 + ty * L::TH, vx0 = tx * kTileW;
  const int wsh = P.wsh, sws = P.sws, RO = kTileW + 2 * wsh, ROH = L::TH + 2 * wsh;
  float4* sCo = smem4;
  float4* sCo2 = sCo + RO * ROH;  // 8-plane input only
  float* sLut = reinterpret_cast<float*>(sCo + (FULL8 ? 2 : 1) * RO * ROH);
  int2* sOff = reinterpret_cast<int2*>(sLut + NPX * kLutWords);

  // the original covariance of the tile and the window's halo; frame rows end
  // at tiles of P.tile_h rows, so the last rows are clamped (outputs that
  // exist never use a clamped one)
  {
    const int Hp = S.tiles_y * P.tile_h + 2 * P.G;
    for (int r = warp; r < ROH; r += L::WARPS) {
      const size_t row = (size_t)min(vy0 - wsh + P.G + r, Hp - 1) * S.pitch + (vx0 - wsh + P.G);
      for (int c = lane; c < RO; c += 32) {
        cp_async16(sCo + r * RO + c, S.cori + row + c);
        if (FULL8) cp_async16(sCo2 + r * RO + c, S.cori2 + row + c);
      }
    }
  }
  // offset t of the window without its centre: the word's place relative to
  // the pixel's in the volume of a pass, and the neighbour's in the tile
  const int nhalf = P.n_off / 2;
  const int plane = G.rows * G.pitch;
  for (int t = tid; t < P.n_off; t += L::THREADS) {
    const int v = t < nhalf ? t : t + 1;
    const int dy = v / sws - wsh, dx = v - (v / sws) * sws - wsh;
    sOff[t] = make_int2(t < nhalf ? (nhalf - 1 - t) * plane + dy * G.pitch + dx : (t - nhalf) * plane, dy * RO + dx);
  }
  cp_async_wait_all();
  __syncthreads();

  const int y0 = warp * PX;
  const int ci = (y0 + wsh) * RO + lane + wsh;
  // pixels past the last virtual row and column repeat it: their words exist
  const int wy = min(vy0 + y0, S.vH) - G.row0, wx = min(vx0 + lane, S.vW) + wsh;
  const int wpitch = vy0 + y0 < S.vH ? G.pitch : 0;
  const uint32_t* words = vol + G.vol + (size_t)wy * G.pitch + wx;

  Best<PX, NM> best;
#pragma unroll
  for (int i = 0; i < PX; ++i) {
    best.e[i] = -1.0f;
    best.rank[i] = 0x7fffffff;
    best.combo[i] = -1;
    best.a[i] = 0.f;
    best.s0[i] = 1.f;
#pragma unroll
    for (int d = 0; d < NM; ++d) best.m[i][d] = 0.f;
  }
  for (int ps = 0; ps < P.npass; ++ps) {
    const PassParams& pp = P.pass[ps];
    const uint32_t* w = words + (size_t)ps * nhalf * plane;
    if (NPX == 1 || pp.np == 1) {
      mean_pass<1, FULL8>(P, pp, w, wpitch, sCo, sCo2, sLut, sOff, RO, ci, best);
    } else if (pp.np == 2) {
      if constexpr (NPX >= 2) mean_pass<2, FULL8>(P, pp, w, wpitch, sCo, sCo2, sLut, sOff, RO, ci, best);
    } else {
      if constexpr (NPX >= 3) mean_pass<3, FULL8>(P, pp, w, wpitch, sCo, sCo2, sLut, sOff, RO, ci, best);
    }
  }
#pragma unroll
  for (int i = 0; i < PX; ++i) {
    const int vy = vy0 + y0 + i, vx = vx0 + lane;
    const int oy = (vy < S.H - 1) ? vy : (vy == S.vH ? S.H - 1 : -1);
    const int ox = (vx < S.W - 1) ? vx : (vx == S.vW ? S.W - 1 : -1);
    if (oy < 0 || ox < 0 || vy >= G.vy1) continue;
    const int o = ci + i * RO;
    float4 c2 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (FULL8) c2 = sCo2[o];
    write_pixel<FULL8>(S, (size_t)oy * S.W + ox, sCo[o], c2, i, best);
  }
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------

// pass shapes with an index kernel: 0 {1,2,3}, 1 {4,5}, 2..6 the single
// halves 1..5; -1 none
int pass_shape(const PassParams& p) {
  if (p.np == 3 && p.ph[0] == 1 && p.ph[1] == 2 && p.ph[2] == 3) return 0;
  if (p.np == 2 && p.ph[0] == 4 && p.ph[1] == 5) return 1;
  if (p.np == 1 && p.ph[0] >= 1 && p.ph[0] <= 5) return 1 + p.ph[0];
  return -1;
}
int shape_phm(int shape) { return shape == 0 ? 3 : (shape == 1 ? 5 : shape - 1); }
int shape_vc(int shape) { return 128 - 8 * ((shape_phm(shape) + 3) / 4); }

template <int PH0, int PH1, int PH2>
cudaError_t launch_index_t(const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                           const PassList& passes, int slot, uint32_t* vol, dim3 grid, size_t smem,
                           cudaStream_t st) {
  static size_t allowed[kMaxDevices];
  const cudaError_t e = allow_dynamic_smem((const void*)nlsar_index_kernel<PH0, PH1, PH2>, smem, allowed);
  if (e != cudaSuccess) return e;
  nlsar_index_kernel<PH0, PH1, PH2><<<grid, kIdxThreads, smem, st>>>(F, scenes, segs, nseg, passes, slot, vol);
  return cudaGetLastError();
}

template <int NPX, bool FULL8>
cudaError_t launch_mean_t(const FilterParams& F, const SceneDesc* scenes, const SplitSeg* segs, int nseg,
                          const uint32_t* vol, int tiles, cudaStream_t st) {
  static size_t allowed[kMaxDevices];
  const size_t smem = mean_smem(F.wsh, NPX, FULL8, F.n_off);
  const cudaError_t e = allow_dynamic_smem((const void*)nlsar_mean_kernel<NPX, FULL8>, smem, allowed);
  if (e != cudaSuccess) return e;
  nlsar_mean_kernel<NPX, FULL8><<<tiles, MeanL<FULL8>::THREADS, smem, st>>>(F, scenes, segs, nseg, vol);
  return cudaGetLastError();
}

int div_up(int a, int b) { return (a + b - 1) / b; }

}  // namespace

bool split_supported(const FilterParams& F, bool full8) {
  return F.prec == 0 && !F.withhold_staging && fast_kernel_supported(F, full8);
}

// Cuts the jobs (row ranges of scenes) into segments of at most `budget`
// words of volume, groups the segments into chunks of at most that size, and
// chooses every chunk's block rows and offset groups.  False where the scene
// is too wide for one tile row's volume.
bool split_layout(const Plan& pl, const std::vector<SceneGeom>& geo, const std::vector<SplitJob>& jobs,
                  size_t budget, int sms, SplitLayout& out) {
  const FilterParams& F = pl.P;
  const int th = pl.full8 ? kSplitTileH8 : kSplitTileH;
  const int nhalf = F.n_off / 2;
  out.segs.clear();
  out.chunks.clear();
  out.vol_words = 0;
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
  size_t used = 0;
  auto close_chunk = [&] {
    if (!out.chunks.empty()) out.chunks.back().seg1 = (int)out.segs.size();
    used = 0;
  };
  for (const SplitJob& j : jobs) {
    const SceneGeom& g = geo[j.scene];
    const int row1 = std::min(j.row1, g.vH + 1);
    if (j.row0 >= row1) continue;
    const int pitch = (g.vW + 1 + 2 * F.wsh + 3) / 4 * 4;
    const size_t row_words = (size_t)F.npass * nhalf * pitch;
    const long long fit = (long long)(budget / row_words) - F.wsh;
    const int most = std::max(th, (int)std::min<long long>(fit, 1 << 20) / th * th);
    const int n = row1 - j.row0;
    const int step = div_up(div_up(n, div_up(n, most)), th) * th;
    for (int y = j.row0; y < row1; y += step) {
      SplitSeg s{};
      s.scene = j.scene;
      s.vy0 = y;
      s.vy1 = std::min(y + step, row1);
      s.row0 = y - F.wsh;
      s.rows = s.vy1 - s.row0;
      s.pitch = pitch;
      s.tiles_x = div_up(g.vW + 1, kTileW);
      // the mean kernel's offsets inside a pass's volume are 32-bit
      if ((size_t)nhalf * s.rows * pitch > 0x7fffffff) return false;
      const size_t words = row_words * s.rows;
      if (out.chunks.empty() || (used && used + words > budget)) {
        close_chunk();
        out.chunks.push_back(SplitChunk{});
        out.chunks.back().seg0 = (int)out.segs.size();
      }
      s.vol = used;
      used += words;
      out.vol_words = std::max(out.vol_words, used);
      out.segs.push_back(s);
    }
  }
  close_chunk();
  for (SplitChunk& c : out.chunks) {
    int tiles = 0;
    for (int i = c.seg0; i < c.seg1; ++i) {
      SplitSeg& s = out.segs[i];
      s.tile_begin = tiles;
      tiles += s.tiles_x * div_up(s.vy1 - s.vy0, th);
    }
    c.tiles = tiles;
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
                         const SceneDesc* d_scenes, const SplitSeg* d_segs, uint32_t* vol, cudaStream_t st) {
  const SplitChunk& c = lay.chunks[chunk];
  const SplitSeg* segs = d_segs + c.seg0;
  const int nseg = c.seg1 - c.seg0;
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < lay.nshape && e == cudaSuccess; ++k) {
    const dim3 grid(c.idx_blocks[k], c.idx_z[k], lay.passes[k].n);
    auto go = [&](auto launch) {
      return launch(F, d_scenes, segs, nseg, lay.passes[k], k, vol, grid, c.idx_smem[k], st);
    };
    switch (lay.shape[k]) {
      case 0: e = go(launch_index_t<1, 2, 3>); break;
      case 1: e = go(launch_index_t<4, 5, -1>); break;
      case 2: e = go(launch_index_t<1, -1, -1>); break;
      case 3: e = go(launch_index_t<2, -1, -1>); break;
      case 4: e = go(launch_index_t<3, -1, -1>); break;
      case 5: e = go(launch_index_t<4, -1, -1>); break;
      case 6: e = go(launch_index_t<5, -1, -1>); break;
      default: e = cudaErrorInvalidValue;
    }
  }
  if (e != cudaSuccess) return e;
  int npx = 1;
  for (int i = 0; i < F.npass; ++i) npx = std::max(npx, F.pass[i].np);
  if (pl.full8)
    return npx == 1 ? launch_mean_t<1, true>(F, d_scenes, segs, nseg, vol, c.tiles, st)
                    : launch_mean_t<3, true>(F, d_scenes, segs, nseg, vol, c.tiles, st);
  return npx == 1 ? launch_mean_t<1, false>(F, d_scenes, segs, nseg, vol, c.tiles, st)
                  : launch_mean_t<3, false>(F, d_scenes, segs, nseg, vol, c.tiles, st);
}

}  // namespace dcl

// From rows of similarities to weight codes: the patch sums and table indices
// of one half-window offset, down a strip of columns (used by the index kernels
// of the two-kernel NL-SAR paths).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "nlsar_common.cuh"
#include "nlsar_math.cuh"

namespace dcl {
namespace {

// A weight's code: one byte, its table entry, or kZeroCode for weight 0
// (d > dmax).  Entry 255 is reached only where the scaled sum rounds to
// exactly 1; it is coded as 254, so a call whose tables have 256 entries needs
// entries 254 and 255 equal (split_tables_ok).
constexpr int kZeroCode = 255;

// The codes of a pass of NP patch sizes at one (offset, pixel).
template <int NP>
struct WordOf {
  using T = uint32_t;
};
template <>
struct WordOf<1> {
  using T = uint8_t;
};
template <>
struct WordOf<2> {
  using T = uint16_t;
};

// Four adjacent words of a lane, stored as one aligned vector.
template <int NP>
__device__ __forceinline__ void store_words(typename WordOf<NP>::T* out, const uint32_t (&w)[4]) {
  if constexpr (NP == 3) {
    *reinterpret_cast<uint4*>(out) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if constexpr (NP == 2) {
    *reinterpret_cast<uint2*>(out) = make_uint2(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410));
  } else {
    *reinterpret_cast<uint32_t*>(out) =
        __byte_perm(__byte_perm(w[0], w[1], 0x0040), __byte_perm(w[2], w[3], 0x0040), 0x5410);
  }
}

// One warp walks down the rows for one offset, each lane owning four adjacent
// columns.  Per row it gets the patch halo from its neighbour lanes by
// shuffles, forms the horizontal sums in nested rings, and keeps, per patch
// size 2 ph + 1, the 2 ph partial vertical sums in flight (the sum of the last
// k rows, top down), so a vertical sum costs 2 ph adds, two columns per packed
// add, and no loads.  A smaller patch is complete PHM - ph rows before the
// largest, so its code waits in `pend`.
// EXACT: the table index as nlsar_kernels.cu takes it, by a rounded division.
template <int PH0, int PH1, int PH2, bool EXACT = false>
struct WordWalk {
  static constexpr int NP = np_of<PH0, PH1, PH2>();
  static constexpr int PHM = cmax(PH0, cmax(PH1, PH2));
  static constexpr int HL = (PHM + 3) / 4;     // lanes at each end of a warp that only supply the halo
  static constexpr int VC = 128 - 8 * HL;      // columns a warp produces
  static constexpr int ND = PHM - PH0;         // rows the first patch's code waits
  static_assert(PH0 >= 1 && 4 * HL >= PHM, "pass shape");

  float inv_span[NP], nbias[NP], lm1[NP], dmax[NP];  // EXACT: the span, the lower end
  float2 vs[NP][2 * PHM][2];  // vs[j][k]: last k + 1 rows of patch j, columns in pairs
  uint32_t pend[ND > 0 ? ND : 1][4];

  // log2_units: the similarities are in log2 units, the lookup scales by ln 2
  __device__ __forceinline__ void set(const FilterParams& P, const PassParams& pp, bool log2_units) {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const ComboParams& cp = P.combo[pp.combo[j]];
      inv_span[j] = EXACT ? cp.span : 1.0f / cp.span;
      nbias[j] = EXACT ? cp.dmin : -cp.dmin * inv_span[j];
      lm1[j] = cp.lm1;
      dmax[j] = cp.dmax;
      if (log2_units) {
        inv_span[j] *= 0.69314718f;
        dmax[j] *= 1.44269504f;
      }
    }
  }

  __device__ __forceinline__ void start() {
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
  }

  // One row: s[PHM .. PHM + 3] are the lane's similarities (the rest is filled
  // here); w the words of the row 2 PHM above.  NAN0: a NaN similarity counts
  // as 0 (else there is none).
  template <bool NAN0>
  __device__ __forceinline__ void row(float (&s)[4 + 2 * PHM], uint32_t (&w)[4]) {
#pragma unroll
    for (int k = 1; k <= PHM; ++k) {
      s[PHM - k] = __shfl_up_sync(0xffffffffu, s[PHM + 3 - (k - 1) % 4], (k + 3) / 4);
      s[PHM + 3 + k] = __shfl_down_sync(0xffffffffu, s[PHM + (k - 1) % 4], (k + 3) / 4);
    }
    float hs[NP][4];
    auto rings = [&] {
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
    };
    rings();
    // the largest rings of the first and last column hold every similarity,
    // so one test finds any NaN
    if (NAN0 && (isnan(hs[NP - 1][0]) || isnan(hs[NP - 1][3]))) {
#pragma unroll
      for (int k = 0; k < 4 + 2 * PHM; ++k)
        if (isnan(s[k])) s[k] = 0.0f;
      rings();
    }
    // vertical sums, the weight's table index
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
        if constexpr (EXACT) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float d = e ? d2.y : d2.x;
            const float dc = fminf(fmaxf(d, nbias[j]), dmax[j]);
            const uint32_t code = (uint32_t)__fmul_rn(__fdiv_rn(__fsub_rn(dc, nbias[j]), inv_span[j]), lm1[j]);
            field[j][2 * q + e] = d > dmax[j] ? (uint32_t)kZeroCode : min(code, (uint32_t)kZeroCode - 1);
          }
          continue;
        }
        // saturating FMA (clamps, NaN to 0), round-toward-zero add of 2^23:
        // the low mantissa bits are the index; d > dmax: weight 0
        const float2 u2 = make_float2(__saturatef(fmaf(d2.x, inv_span[j], nbias[j])),
                                      __saturatef(fmaf(d2.y, inv_span[j], nbias[j])));
        const float2 t2 = __ffma2_rz(u2, make_float2(lm1[j], lm1[j]), make_float2(8388608.0f, 8388608.0f));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t code = min(__float_as_uint(e ? t2.y : t2.x), 0x4B000000u + (kZeroCode - 1));
          field[j][2 * q + e] = (e ? d2.y : d2.x) > dmax[j] ? (uint32_t)kZeroCode : code;  // the low byte counts
        }
      }
    }
    // byte j of a word is the code of patch j
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      uint32_t next = 0;
#pragma unroll
      for (int k = ND; k >= 0; --k) {  // rows waited, the smallest patch first
        uint32_t v = k < ND ? pend[k][o] : 0u;
#pragma unroll
        for (int j = 0; j < NP; ++j)
          if (PHM - ph_of<PH0, PH1, PH2>(j) == k)
            v = j == 0 ? field[0][o] : __byte_perm(v, field[j][o], j == 1 ? 0x0040 : 0x0410);
        if (k < ND) pend[k][o] = next;
        next = v;
      }
      w[o] = next;
    }
  }
};

}  // namespace
}  // namespace dcl

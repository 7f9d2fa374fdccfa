// Device arithmetic shared by the NL-SAR kernels of 2x2 covariances: the GLR
// similarity, the statistics and selection of one (patch, scale) combination,
// and the blended output.  One copy, so that the kernels give the same bits.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "nlsar_common.cuh"

namespace dcl {
namespace {

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }

template <int PH0, int PH1, int PH2>
__host__ __device__ constexpr int np_of() {
  return (PH0 >= 0) + (PH1 >= 0) + (PH2 >= 0);
}

// Arithmetic variants of the similarity and the sums (the precision study;
// kPrecRatio is the default):
//   kPrecRatio  the GLR as one base-2 log of the ratio
//               det(A+B)^2 / (2^4 det A det B) (sim_measures.h:52-64 is the
//               natural log of that ratio), with 1/(4 det) of every staged
//               pixel precomputed; the similarities and patch sums are in
//               log2 units and the weight lookup scales by ln 2.  No large
//               logs cancel, so the similarity keeps about 1e-7 absolute
//               accuracy where the log form loses the ulps of ln det (~1e-6)
//   kPrecLog2   the log form 2 ln det(A+B) - ln det A - ln det B - 4 ln 2 with
//               the per-pixel ln det staged and an approximate base-2 log
//   kPrecLogf   the log form with the correctly rounded logf, the reference's
//               arithmetic
//   kPrecKahan  kPrecRatio with Kahan-compensated patch sums and accumulators
//   kPrecHalf   kPrecRatio with every similarity rounded to FP16, as FP16
//               staging of the similarity map would store it
enum { kPrecRatio = 0, kPrecLog2 = 1, kPrecLogf = 2, kPrecKahan = 3, kPrecHalf = 4 };

template <int PV>
__host__ __device__ constexpr bool ratio_form() {
  return PV == kPrecRatio || PV == kPrecKahan || PV == kPrecHalf;
}

// det of a staged scaled covariance, rounded like the prep kernel's
// (sim_measures.h:31-34)
__device__ __forceinline__ float det_of(const float4 c) {
  return __fsub_rn(__fmul_rn(c.x, c.y), __fadd_rn(__fmul_rn(c.z, c.z), __fmul_rn(c.w, c.w)));
}

// The per-pixel term of a staged pixel: ln det (log forms) or 1/(4 det)
// (ratio form; NaN for a negative det, whose log is NaN, +inf for det 0).
template <int PV>
__device__ __forceinline__ float pixel_term(const float4 c) {
  const float d = det_of(c);
  if (!ratio_form<PV>()) return logf(d);
  return d >= 0.0f ? __fdiv_rn(0.25f, fabsf(d)) : __int_as_float(0x7fffffff);
}

// load of one float from a 32-bit shared-memory address, for tables that
// stay unchanged while they are read (the compiler may schedule it freely)
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

__device__ __forceinline__ float lg2_ftz(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float kahan_add(float s, float x, float& c) {
  const float y = x - c;
  const float t = s + y;
  c = (t - s) - y;
  return t;
}

// det(A + B), with every rounding explicit so that all kernels share it
__device__ __forceinline__ float det_sum(const float4 a, const float4 b) {
  const float2 d01 = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
  const float2 d23 = __fadd2_rn(make_float2(a.z, a.w), make_float2(b.z, b.w));
  return __fmaf_rn(d01.x, d01.y, -__fmaf_rn(d23.x, d23.x, __fmul_rn(d23.y, d23.y)));
}

// The ratio form: log2 of det |det| / (16 det A det B); NaN (the log of a
// negative number) when det < 0
__device__ __forceinline__ float glr_ratio(const float4 a, float la, const float4 b, float lb) {
  const float det = det_sum(a, b);
  return lg2_ftz(__fmul_rn(__fmul_rn(det, fabsf(det)), __fmul_rn(la, lb)));
}

template <int PV>
__device__ __forceinline__ float glr_sim(const float4 a, float la, const float4 b, float lb, float c2d) {
  // sim_measures.h:52-64 with nlooks 1 and the per-pixel terms precomputed;
  // NaN -> 0.  Each form is exactly symmetric in (A, B), which gives the
  // mirrored half window the reference's values (copy_symm_weights.cl:56-76).
  float r;
  if (ratio_form<PV>()) {
    r = glr_ratio(a, la, b, lb);
    if (PV == kPrecHalf) r = __half2float(__float2half_rn(r));
  } else {
    const float det = det_sum(a, b);
    const float t = (la + lb) + c2d;
    r = (PV == kPrecLogf) ? 2.0f * logf(det) - t : fmaf(2.0f * 0.69314718f, __log2f(det), -t);
  }
  if (r != r) r = 0.0f;
  return r;
}

// patch half size of pass component j (compile time)
template <int PH0, int PH1, int PH2>
__device__ __forceinline__ constexpr int ph_of(int j) {
  return j == 0 ? PH0 : (j == 1 ? PH1 : PH2);
}

// Selection state of a thread's PX pixels, kept across the passes.
template <int PX, int NM>
struct Best {
  float e[PX], a[PX], s0[PX], m[PX][NM];
  int rank[PX], combo[PX];
};

// Statistics, alpha, ENL' (compute_nl_statistics.cl:92-101,
// compute_alphas.cl:30-41, compute_enls_nobias.cl:19-22) of one combination
// from its accumulators A = {sum w, w^2, w I0, w I1, w I0^2, w I1^2, w Re C01,
// w Im C01, 8-plane input: four more planes}, and its entry in pixel i's
// selection state (best_params.cpp).
template <int PX, int NM, int NA>
__device__ __forceinline__ void select_combo(const FilterParams& P, int combo, const float (&A)[NA], int i,
                                             Best<PX, NM>& best) {
  const float s0 = A[0], s1 = A[1], s2 = A[2], s3 = A[3], s4 = A[4], s5 = A[5], s6 = A[6], s7 = A[7];
  const float enl = s0 * s0 / s1;
  const float i0 = s2 / s0, i1 = s3 / s0;
  // explicitly rounded, so that no kernel contracts them differently
  const float q0 = __fmul_rn(i0, i0), q1 = __fmul_rn(i1, i1);
  const float v0 = __fsub_rn(s4 / s0, q0), v1 = __fsub_rn(s5 / s0, q1);
  float alpha = 0.0f;
  alpha = fmaxf(alpha, fmaxf(0.0f, __fsub_rn(v0, q0) / v0));
  alpha = fmaxf(alpha, fmaxf(0.0f, __fsub_rn(v1, q1) / v1));
  if (P.alpha_zero) alpha = 0.0f;
  const float oma = 1.0f - alpha;
  const float enb = enl / (oma * oma + (alpha * alpha + 2.0f * alpha * (1.0f - alpha) / s0) * enl);
  const int rank = P.combo[combo].rank;
  const bool take = (P.select_mode == 0) || (enb > best.e[i]) || (enb == best.e[i] && rank < best.rank[i]);
  const bool take_fb = !take && best.combo[i] < 0 && combo == P.fallback_combo;
  if (take) {
    best.e[i] = enb;
    best.rank[i] = rank;
  }
  if (take || take_fb) {
    best.combo[i] = combo;
    best.a[i] = alpha;
    best.s0[i] = s0;
    best.m[i][0] = s2;
    best.m[i][1] = s3;
    best.m[i][2] = s6;
    best.m[i][3] = s7;
#pragma unroll
    for (int e = 4; e < NM; ++e) best.m[i][e] = A[(e + 4) % NA];
  }
}

// The blend with the centre (weighted_means.cl:79) of pixel i, written to
// output o: InSAR input decomposed (covmat_decompose.cl:32-37), 8-plane input
// as its planes (c2 = {Im C00, Re C10, Im C10, Im C11} of the centre).
template <bool FULL8, int PX, int NM>
__device__ __forceinline__ void write_pixel(const SceneDesc& S, size_t o, const float4 c, const float4 c2, int i,
                                            const Best<PX, NM>& best) {
  const float alpha = best.a[i], s0 = best.s0[i];
  const float oma = 1.0f - alpha;
  const float c00 = oma * best.m[i][0] / s0 + alpha * c.x;
  const float c11 = oma * best.m[i][1] / s0 + alpha * c.y;
  const float cre = oma * best.m[i][2] / s0 + alpha * c.z;
  const float cim = oma * best.m[i][3] / s0 + alpha * c.w;
  if (FULL8) {
    // planes {Re, Im} of C00, C01, C10, C11
    const size_t n = (size_t)S.H * S.W;
    S.cov_out[o] = c00;
    S.cov_out[n + o] = oma * best.m[i][4 % NM] / s0 + alpha * c2.x;
    S.cov_out[2 * n + o] = cre;
    S.cov_out[3 * n + o] = cim;
    S.cov_out[4 * n + o] = oma * best.m[i][5 % NM] / s0 + alpha * c2.y;
    S.cov_out[5 * n + o] = oma * best.m[i][6 % NM] / s0 + alpha * c2.z;
    S.cov_out[6 * n + o] = c11;
    S.cov_out[7 * n + o] = oma * best.m[i][7 % NM] / s0 + alpha * c2.w;
  } else {
    const float am = sqrtf(c00), as = sqrtf(c11);
    const float r = 0.5f * (am + as);
    S.ref[o] = r * r;
    S.phase[o] = atan2f(cim, cre);
    S.coh[o] = sqrtf(cim * cim + cre * cre) / (am * as);
  }
  if (S.sel_out) S.sel_out[o] = best.combo[i];
}

}  // namespace
}  // namespace dcl

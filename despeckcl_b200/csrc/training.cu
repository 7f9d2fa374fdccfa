// NL-SAR training on the GPU: dissimilarities of every pair of patches of a
// homogeneous area and the quantile / chi-squared LUTs, for 2x2 and 3x3
// covariances.
//
// Follows (paths relative to the despeckCL project root):
//   src/compute/nlsar/training/get_stats.cpp:25-59      one entry per (patch, scale), lut_size 256
//   src/compute/nlsar/training/get_dissims.cpp:32-117   rescale, Gaussian average with s_max = s
//   src/compute/nlsar/training/patches.cpp:32-136       non-overlapping p x p patches from (0,0),
//                                                       clamp-padded at the far edges; dissimilarity
//                                                       = sum over the p*p pixels of the GLR measure,
//                                                       later patch first
//   src/compute/nlsar/training/combinations.cpp:26-41   every unordered pair
//   src/compute/nlsar/stats.cpp:28-80                   LUTs
//
// The LUT of a combination needs the extremes of its dissimilarities and how
// many lie below each of 256 thresholds between them, not their order: the
// pairs kernel reduces the extremes, a second pass counts, and one copy of all
// combinations' counts comes back.  (Sorting 1.7 million values per
// combination and filtering them on the host, with device allocations per
// combination, took 17 ms for a 128 x 128 area and six combinations.)

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/despeckcl_b200.h"
#include "dcl_internal.h"
#include "nlsar_common.cuh"
#include "nlsar_split3.cuh"
#include "stats_internal.h"

namespace dcl {

std::vector<float> gauss_weights(int s);
float rescale_gamma_2x2();

namespace {

constexpr int kLut = 256;  // get_stats.cpp:31

// Buffers up to this size come from the stream-ordered pool, which keeps them;
// larger ones (a 128 x 128 area in 1 x 1 patches has 0.5 GiB of pairs, 300 x 300
// 15 GiB) go back to the device after the call.
constexpr size_t kTrainPoolBytes = size_t(256) << 20;

// What one combination's LUT is made of.  The extremes as order-preserving
// keys (lo inverted, so that zeroed memory is empty).
struct LutCounts {
  unsigned lo_inv, hi;
  unsigned long long finite;
  unsigned long long bins[kLut + 1];  // bins[b]: values with exactly b thresholds at or below them
};

__device__ __forceinline__ unsigned key_of(float v) {
  const unsigned b = __float_as_uint(v);
  return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__host__ __device__ __forceinline__ unsigned bits_of_key(unsigned k) { return k & 0x80000000u ? k & 0x7fffffffu : ~k; }

__global__ void train_cov_insar_kernel(const float* __restrict__ a1, const float* __restrict__ a2,
                                       const float* __restrict__ phi, size_t n, float* __restrict__ cov) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // src/data/data.cpp:70-88
  const float am = a1[i], as = a2[i];
  float sn, cs;
  sincosf(phi[i], &sn, &cs);
  cov[i] = am * am;
  cov[n + i] = as * as;
  cov[2 * n + i] = am * as * cs;
  cov[3 * n + i] = am * as * sn;
}

// Plane of similarity real k (diagonal first, then Re and Im of the upper
// triangle) among the input planes.
struct TrainPlanes {
  int at[9];
};

__device__ __forceinline__ float det_q(const float (&a)[4]) { return (a[0] * a[1]) - (a[2] * a[2] + a[3] * a[3]); }
__device__ __forceinline__ float det_q(const float (&a)[9]) { return det3f(a); }

// Q similarity reals (4: 2x2, 9: 3x3), rescaled (covmat_rescale.cl:31-39) and
// averaged (covmat_spatial_avg.cl:50-57, s_max = s) on the valid region (H-s+1)
// x (W-s+1), of every patch pixel, and their ln det, laid out [real][pixel of
// the patch][patch]; patch k at ((k / nw) * p, (k % nw) * p), clamp padding
// (src/data/sub_images.cpp:37-38)
template <int Q>
__global__ void train_patches_kernel(const float* __restrict__ cov, TrainPlanes pl, int H, int W, int s, GaussArg ga,
                                     float gamma, int p, int nw, int n, float* __restrict__ patches) {
  constexpr int D = Q == 4 ? 2 : 3;  // diagonal reals
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int pp = p * p;
  if (i >= n * pp) return;
  const int r = i / n, k = i - r * n;
  const int y = min(H - s, (k / nw) * p + r / p);
  const int x = min(W - s, (k % nw) * p + r % p);
  const size_t plane = (size_t)H * W;
  float a[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) a[q] = 0.0f;
  for (int kx = 0; kx < s; ++kx)
    for (int ky = 0; ky < s; ++ky) {
      const size_t at = (size_t)(y + kx) * W + x + ky;
      const float g = ga.g[kx * s + ky];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float v = cov[pl.at[q] * plane + at];
        a[q] = fmaf(g, q >= D ? v * gamma : v, a[q]);
      }
    }
  const size_t stride = (size_t)n * pp;
#pragma unroll
  for (int q = 0; q < Q; ++q) patches[q * stride + i] = a[q];
  patches[Q * stride + i] = logf(det_q(a));
}

constexpr int kPairThreads = 128;

// Pairs (hi, j), hi > j: a block takes 128 consecutive j and `rows` hi, so its
// loads of patch j are coalesced and those of patch hi uniform.  A thread's
// chain of logarithms is what a small area waits for, so the caller takes few
// rows where the blocks are few.
template <int Q>
__global__ void __launch_bounds__(kPairThreads)
    train_pairs_kernel(const float* __restrict__ patches, int pp, int n, int rows, float c2d,
                       float* __restrict__ out, LutCounts* __restrict__ lut) {
  const int j = blockIdx.x * kPairThreads + threadIdx.x;
  const int hi0 = blockIdx.y * rows, hi1 = min(hi0 + rows, n);
  if (hi1 - 1 <= blockIdx.x * kPairThreads) return;  // no hi above the block's first j
  const size_t stride = (size_t)n * pp;
  const float* B = patches + j;
  unsigned lo_inv = 0, top = 0, finite = 0;
  for (int hi = hi0; hi < hi1; ++hi) {
    if (j >= hi) continue;
    const float* A = patches + hi;
    float sum = 0.0f;
#pragma unroll 4
    for (int i = 0; i < pp; ++i) {
      // sim_measures.h:37-65, 100-160 with nlooks 1: first argument a, second b
      float s[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) s[q] = A[q * stride + (size_t)i * n] + B[q * stride + (size_t)i * n];
      const float la = A[Q * stride + (size_t)i * n], lb = B[Q * stride + (size_t)i * n];
      float r = -(c2d + la + lb - 2.0f * logf(det_q(s)));
      if (r != r) r = 0.0f;
      sum += r;
    }
    out[(long long)hi * (hi - 1) / 2 + j] = sum;
    if (isfinite(sum)) {  // stats.cpp:28-38 drops NaN and inf
      const unsigned k = key_of(sum);
      lo_inv = max(lo_inv, ~k);
      top = max(top, k);
      ++finite;
    }
  }
  lo_inv = __reduce_max_sync(0xffffffffu, lo_inv);
  top = __reduce_max_sync(0xffffffffu, top);
  finite = __reduce_add_sync(0xffffffffu, finite);
  if ((threadIdx.x & 31) == 0 && finite) {
    atomicMax(&lut->lo_inv, lo_inv);
    atomicMax(&lut->hi, top);
    atomicAdd(&lut->finite, (unsigned long long)finite);
  }
}

// Counts the values between consecutive thresholds dmin + i step
// (stats.cpp:45-52; each product and sum rounded as on the host).
__global__ void __launch_bounds__(256)
    train_count_kernel(const float* __restrict__ dis, long long npairs, LutCounts* __restrict__ lut) {
  __shared__ unsigned hist[kLut + 1];
  for (int i = threadIdx.x; i <= kLut; i += 256) hist[i] = 0;
  __syncthreads();
  const float dmin = __uint_as_float(bits_of_key(~lut->lo_inv)), dmax = __uint_as_float(bits_of_key(lut->hi));
  const float step = __fdiv_rn(__fsub_rn(dmax, dmin), (float)kLut);
  const float inv = step > 0.0f ? 1.0f / step : 0.0f;
  auto threshold = [&](int i) { return __fadd_rn(dmin, __fmul_rn((float)i, step)); };
  for (long long t = (long long)blockIdx.x * 256 + threadIdx.x; t < npairs; t += (long long)gridDim.x * 256) {
    const float d = dis[t];
    if (!isfinite(d)) continue;
    // thresholds are non-decreasing: a guess, corrected to the exact number
    // at or below d
    int b = max(0, min(kLut, __float2int_rd((d - dmin) * inv) + 1));
    while (b < kLut && threshold(b) <= d) ++b;
    while (b > 0 && threshold(b - 1) > d) --b;
    atomicAdd(&hist[b], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= kLut; i += 256)
    if (hist[i]) atomicAdd(&lut->bins[i], (unsigned long long)hist[i]);
}

// One (patch, scale) combination of a training call.
struct TrainCombo {
  int p, s, nw;
  long long n, npairs;
};

int train_combos(int H, int W, const int* patches, int np, const int* scales, int ns, std::vector<TrainCombo>& out) {
  if (!patches || !scales || np < 1 || ns < 1)
    return set_error(DCL_ERR_INVALID_ARGUMENT, "patch_sizes and scale_sizes must not be empty");
  // get_stats.cpp:33-37: patch outer, scale inner
  for (int pi = 0; pi < np; ++pi)
    for (int si = 0; si < ns; ++si) {
      TrainCombo c;
      c.p = patches[pi];
      c.s = scales[si];
      if (c.p < 1 || c.p % 2 == 0 || c.s < 1 || c.s % 2 == 0 || c.s * c.s > kMaxGauss)
        return set_error(DCL_ERR_INVALID_ARGUMENT, "patch and scale sizes must be odd (scale <= 9)");
      const int Ho = H - c.s + 1, Wo = W - c.s + 1;
      if (Ho < 1 || Wo < 1)
        return set_error(DCL_ERR_INVALID_ARGUMENT, "training area %dx%d smaller than scale %d", H, W, c.s);
      c.nw = (Wo + c.p - 1) / c.p;
      c.n = (long long)((Ho + c.p - 1) / c.p) * c.nw;
      if (c.n < 2)
        return set_error(DCL_ERR_INVALID_ARGUMENT, "training area holds fewer than two %dx%d patches", c.p, c.p);
      if (c.n * c.p * c.p > 0x7fffffff) return set_error(DCL_ERR_INVALID_ARGUMENT, "training area too large");
      c.npairs = c.n * (c.n - 1) / 2;
      out.push_back(c);
    }
  return DCL_OK;
}

// Trains every combination on `nplane` host planes of H x W: the covariance's
// (Q 4: eight, Q 9: eighteen) or, with `insar`, the two amplitudes and the
// phase.  Null on failure.
template <int Q>
dcl_stats_collection* train(const float* const* planes, int nplane, bool insar, const TrainPlanes& where, float gamma,
                            float c2d, int H, int W, const int* patches, int np, const int* scales, int ns) {
  std::vector<TrainCombo> combos;
  int dev = 0;
  if (train_combos(H, W, patches, np, scales, ns, combos) != DCL_OK || ensure_device_ready(dev) != DCL_OK)
    return nullptr;
  const size_t n = (size_t)H * W;
  const size_t ncov = n * (insar ? 3 + Q : nplane);
  size_t npat = 0, ndis = 0;
  for (const TrainCombo& c : combos) {
    npat = std::max(npat, (size_t)((Q + 1) * c.n * c.p * c.p));
    ndis = std::max(ndis, (size_t)c.npairs);
  }
  const size_t lut_bytes = combos.size() * sizeof(LutCounts);
  cudaStream_t st = cudaStreamPerThread;
  char* mem = nullptr;
  const size_t bytes = lut_bytes + (ncov + npat + ndis) * sizeof(float);
  const bool pooled = bytes <= kTrainPoolBytes;
  cudaError_t e = pooled ? cudaMallocAsync(&mem, bytes, st) : cudaMalloc(&mem, bytes);
  if (e != cudaSuccess) {
    cuda_error(e, "training buffers");
    return nullptr;
  }
  LutCounts* d_lut = reinterpret_cast<LutCounts*>(mem);
  float* d_in = reinterpret_cast<float*>(mem + lut_bytes);
  float* d_cov = insar ? d_in + 3 * n : d_in;
  float* d_pat = d_in + ncov;
  float* d_dis = d_pat + npat;
  e = cudaMemsetAsync(d_lut, 0, lut_bytes, st);
  for (int i = 0; i < nplane && e == cudaSuccess; ++i)
    e = cudaMemcpyAsync(d_in + i * n, planes[i], n * sizeof(float), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && insar)
    train_cov_insar_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d_in, d_in + n, d_in + 2 * n, n, d_cov);
  const int sms = sm_count(dev);
  for (size_t i = 0; i < combos.size() && e == cudaSuccess; ++i) {
    const TrainCombo& c = combos[i];
    GaussArg ga;
    std::memset(&ga, 0, sizeof ga);
    const std::vector<float> g = gauss_weights(c.s);
    std::copy(g.begin(), g.end(), ga.g);
    const int pp = c.p * c.p, nn = (int)c.n;
    train_patches_kernel<Q><<<(unsigned)((c.n * pp + 127) / 128), 128, 0, st>>>(d_cov, where, H, W, c.s, ga, gamma,
                                                                              c.p, c.nw, nn, d_pat);
    const int gx = (nn + kPairThreads - 1) / kPairThreads;
    int rows = 16;
    while (rows > 1 && (long long)gx * ((nn + rows - 1) / rows) < 8LL * sms) rows /= 2;
    train_pairs_kernel<Q><<<dim3(gx, (nn + rows - 1) / rows), kPairThreads, 0, st>>>(d_pat, pp, nn, rows, c2d, d_dis,
                                                                                   d_lut + i);
    train_count_kernel<<<(unsigned)std::min<long long>((c.npairs + 1023) / 1024, 8LL * sms), 256, 0, st>>>(
        d_dis, c.npairs, d_lut + i);
    e = cudaGetLastError();
  }
  profile_count((insar ? 1 : 0) + 3 * (int)combos.size());
  // the chi-squared table is the same for every combination; the host makes it
  // while the device works
  const std::vector<float> chi2 = chi2_table(kLut);
  std::vector<LutCounts> lut(combos.size());
  if (e == cudaSuccess) e = cudaMemcpyAsync(lut.data(), d_lut, lut_bytes, cudaMemcpyDeviceToHost, st);
  if (pooled) cudaFreeAsync(mem, st);
  const cudaError_t e2 = cudaStreamSynchronize(st);
  if (!pooled) cudaFree(mem);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) {
    cuda_error(e, "training");
    return nullptr;
  }
  dcl_stats_collection* out = dcl_collection_new();
  for (size_t i = 0; i < combos.size(); ++i) {
    const LutCounts& l = lut[i];
    if (l.finite == 0) {
      set_error(DCL_ERR_INVALID_ARGUMENT, "no finite dissimilarity in the training area");
      dcl_stats_collection_free(out);
      return nullptr;
    }
    OwnedStats s;
    s.lut_size = kLut;
    const unsigned lo = bits_of_key(~l.lo_inv), hi = bits_of_key(l.hi);
    std::memcpy(&s.dmin, &lo, sizeof lo);
    std::memcpy(&s.dmax, &hi, sizeof hi);
    // the share of values below threshold i: those with at most i thresholds
    // at or below them (stats.cpp:45-58)
    unsigned long long below = 0;
    s.quant.resize(kLut);
    for (int k = 0; k < kLut; ++k) {
      below += l.bins[k];
      s.quant[k] = (float)below / (float)l.finite;
    }
    s.chi2 = chi2;
    dcl_collection_put(out, combos[i].p, combos[i].s, std::move(s));
  }
  return out;
}

float rescale_gamma_3x3() {
  // covmat_rescale.cl:25-26 with nlooks = 1, dimension = 3
  return std::pow(std::min(1.0f / 3.0f, 1.0f), 0.33333f);
}

}  // namespace
}  // namespace dcl

using namespace dcl;

extern "C" dcl_stats_collection* dcl_nlsar_training_insar(const float* a1, const float* a2, const float* phi, int H,
                                                          int W, const int* patches, int np, const int* scales,
                                                          int ns) {
  if (!a1 || !a2 || !phi || H < 1 || W < 1) {
    set_error(DCL_ERR_INVALID_ARGUMENT, "null input or empty training area");
    return nullptr;
  }
  const float* in[3] = {a1, a2, phi};
  return train<4>(in, 3, true, TrainPlanes{{0, 1, 2, 3}}, rescale_gamma_2x2(), 2 * 2 * std::log(2.0f), H, W, patches,
                  np, scales, ns);
}

extern "C" dcl_stats_collection* dcl_nlsar_training_covmat(const float* cov, int H, int W, int dim,
                                                           const int* patches, int np, const int* scales, int ns) {
  if (dim != 2 && dim != 3) {
    set_error(DCL_ERR_INVALID_ARGUMENT, "covariance dimension %d: 2x2 and 3x3 covariances are supported", dim);
    return nullptr;
  }
  if (!cov || H < 1 || W < 1) {
    set_error(DCL_ERR_INVALID_ARGUMENT, "null input or empty training area");
    return nullptr;
  }
  const float* in[18];
  for (int p = 0; p < 2 * dim * dim; ++p) in[p] = cov + (size_t)p * H * W;
  if (dim == 2)
    return train<4>(in, 8, false, TrainPlanes{{0, 6, 2, 3}}, rescale_gamma_2x2(), 2 * 2 * std::log(2.0f), H, W,
                    patches, np, scales, ns);
  TrainPlanes where;
  for (int k = 0; k < 9; ++k) where.at[k] = sim_plane(k);
  return train<9>(in, 18, false, where, rescale_gamma_3x3(), 2 * 3 * std::log(2.0f), H, W, patches, np, scales, ns);
}

// NL-InSAR (despeckcl::nlinsar, src/compute/nlinsar/nlinsar.cpp:42-130 and
// nlinsar_sub_image.cpp:32-250 in the reference).
//
// niter passes; each pass cuts the scene into the reference's 80 x 80 tiles
// with overlap wsh + psh (tile_iterator.cpp, clamped gather sub_images.cpp),
// filters every tile from the previous pass's estimates, and takes each output
// pixel from the tile that writes it last in the reference's clamped
// write-back (tile row y / step for y < H-1, the last tile row's last centre
// row for y = H-1; columns alike).  Three kernels:
//
//  nlinsar_filter_values_kernel  once per call: 0.5 (a1^2 + a2^2) and
//      a1 a2 e^{-j phi} per pixel (precompute_filter_values.cl);
//  nlinsar_weights_kernel  one CTA per tile and group of offsets, the tile's
//      planes in shared memory; per search-window offset: the pixel similarity
//      and the Kullback-Leibler divergence of the estimates (sim_measures.h) on
//      the similarity grid -- with the two pixels swapped in the tile interior
//      for the first wsh window rows, which the reference copies from the
//      mirrored offset (precompute_similarities_{1st,2nd}_pass): each lower-row
//      offset is taken with its mirror, whose interior maps are the lower
//      offset's shifted, only its border evaluated --, p x p sums rows
//      first (precompute_patch_similarities.cl), w = exp(S/h + KL/T) with
//      NaN / inf -> 0 and the centre weight 0 (compute_weights.cl); weights go
//      to a scratch [tile][offset][pixel].  The similarities do not depend on
//      the estimates: a call of several passes keeps the first one's patch sums
//      S (in a second scratch of that shape) and evaluates only divergences
//      after it; divergences from all-zero estimates are zero and skipped;
//  nlinsar_estimate_kernel  one thread per tile pixel that owns its output:
//      the looks (sum w)^2 / sum w^2 in the order the offsets are taken
//      (compute_number_of_looks.cl); below lmin looks the lmin largest weights among the window pixels whose
//      master amplitude is below twice the centre's become their mean, chosen
//      with the reference's std::priority_queue (smoothing.cpp:65-117, a binary
//      heap replayed exactly); then the weighted means (compute_insar.cl),
//      each estimate kept from the previous pass where not finite or 0.
// This file is compiled with -fmad=false: every sum and product is rounded as
// in the reference's kernels; only the math functions (pow, asin, log, exp,
// cos, sin, atan2) are CUDA's.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/despeckcl_b200.h"
#include "dcl_internal.h"

namespace dcl {
namespace {

constexpr int kTile = 80;        // nlinsar.cpp:84, tile_dims {80, 80}
// Threads of the weights kernel: with the similarity maps one CTA fills an
// SM's shared memory; the divergence maps alone leave room for two, whose
// barriers then cover each other.
__host__ __device__ constexpr int weights_threads(bool sim) { return sim ? 1024 : 512; }
constexpr int kMaxLmin = 64;
constexpr int kEstThreads = 128;
constexpr size_t kWeightsBytes = size_t(4) << 30;  // weights held at a time

struct NlGeom {
  int H, W, sws, wsh, p, psh, ov;
  int hsim, hori;      // similarity grid and output side of a tile
  int step;            // tile origin step, kTile - 2 ov
  int ntx, nty;        // tiles per row / column
  int lmin;
  float h, T;
  int nborder;         // similarity-grid positions outside the interior the reference copies
  int mirror;          // 1: offsets of the lower window rows share their maps with their mirrors
};

__device__ __forceinline__ int clampn(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// sim_measures.h:27-40 (am/as/dp of pixel 1, then of pixel 2)
__device__ __forceinline__ float pixel_sim(float am1, float as1, float dp1, float am2, float as2, float dp2) {
  const float s = am1 * am1 + as1 * as1 + am2 * am2 + as2 * as2;
  const float A = s * s;
  const float B = 4.0f * (am1 * am1 * as1 * as1 + am2 * am2 * as2 * as2 + 2.0f * am1 * as1 * am2 * as2 * cosf(dp1 - dp2));
  const float C = am1 * as1 * am2 * as2;
  // pow(x, 1.5) as x sqrt(x) (the same value up to rounding, NaN for x < 0
  // as pow gives) and the hardware log below (a few ulps): 8 % of the pass,
  // with every tested pixel still within tolerance of the oracle; fast
  // divisions or the hardware cos cost agreement
  const float x = C / B;
  const float f = (x * sqrtf(x)) * ((A + B) / A * sqrtf(B / (A - B)) - asinf(sqrtf(B / A)));
  if (f == 0.0f || isnan(f)) return 0.0f;
  return __logf(f);
}

// sim_measures.h:42-50, OpenCL's float pi
__device__ __forceinline__ float pixel_kl(float r1, float d1, float c1, float r2, float d2, float c2) {
  const float cs = cosf(d1 - d2);
  const float a1 = (r2 != 0.0f) ? r1 / r2 * (1.0f - c1 * c2 * cs) / (1.0f - c2 * c2) : 1.0f;
  const float a2 = (r2 != 0.0f) ? r2 / r1 * (1.0f - c1 * c2 * cs) / (1.0f - c1 * c1) : 1.0f;
  return -4.0f / 3.14159274101257324f * (a1 + a2 - 2.0f);
}

__global__ void nlinsar_filter_values_kernel(const float* __restrict__ a1, const float* __restrict__ a2,
                                             const float* __restrict__ dp, float* __restrict__ fa,
                                             float* __restrict__ fr, float* __restrict__ fi, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x1 = a1[i], x2 = a2[i], d = dp[i];
  fa[i] = 0.5f * (x1 * x1 + x2 * x2);
  fr[i] = x1 * x2 * cosf(-d);
  fi[i] = x1 * x2 * sinf(-d);
}

// Sizes of a tile's maps: compile-time for the usual search windows and patch
// sizes (the maps' index divisions become multiplications), else from the call.
template <int SWS_, int P_>
struct NlSizes {
  static constexpr bool FIXED = SWS_ > 0;
  const NlGeom& g;
  __device__ __forceinline__ int sws() const { return FIXED ? SWS_ : g.sws; }
  __device__ __forceinline__ int wsh() const { return FIXED ? (SWS_ - 1) / 2 : g.wsh; }
  __device__ __forceinline__ int p() const { return FIXED ? P_ : g.p; }
  __device__ __forceinline__ int hsim() const { return FIXED ? kTile - SWS_ + 1 : g.hsim; }
  __device__ __forceinline__ int hori() const { return FIXED ? kTile - (SWS_ - 1) - (P_ - 1) : g.hori; }
  __device__ __forceinline__ int nborder() const {
    return FIXED ? wsh() * hsim() + (hsim() - wsh()) * 2 * wsh() : g.nborder;
  }
};

// Work of a tile in units, in the order the looks sum their weights: with
// mirrored maps the offsets of the centre window row, then every lower-row
// offset with its mirror; else every offset.
constexpr float kPairCost = 1.6f;  // a pair of mirrored offsets, in single offsets

__host__ __device__ inline int nl_units(const NlGeom& g) { return g.mirror ? g.sws + g.wsh * g.sws : g.sws * g.sws; }
// first unit of group z of Z groups of about equal cost
__host__ __device__ inline int nl_group(const NlGeom& g, int z, int Z) {
  if (!g.mirror) return (int)((long long)nl_units(g) * z / Z);
  const float at = (g.sws + kPairCost * (g.wsh * g.sws)) * z / Z;
  const int u = at <= g.sws ? (int)at : g.sws + (int)((at - g.sws) / kPairCost);
  return z == Z ? nl_units(g) : (u < nl_units(g) ? u : nl_units(g));
}

// SIM: evaluate similarities (else their patch sums, over h, are read from
// `sums`).
template <class Z_, bool SIM>
__global__ void __launch_bounds__(weights_threads(SIM), SIM ? 1 : 2)
    nlinsar_weights_kernel(const float* __restrict__ a1, const float* __restrict__ a2, const float* __restrict__ dp,
                           const float* __restrict__ rf, const float* __restrict__ pf, const float* __restrict__ cf,
                           const __grid_constant__ NlGeom g, int tile0, const int* __restrict__ nonzero,
                           float* __restrict__ sums, float* __restrict__ wout) {
  extern __shared__ float sm[];
  constexpr int kThreads = weights_threads(SIM);
  const Z_ z{g};
  constexpr int n2 = kTile * kTile;
  float* sRf = sm;
  float* sPf = sRf + n2;
  float* sCf = sPf + n2;
  float* sA1 = sCf + n2;  // SIM only: the amplitudes and the phase
  float* sA2 = sA1 + n2;
  float* sDp = sA2 + n2;
  const int nsim = z.hsim() * z.hsim(), npix = z.hori() * z.hori(), nrow = z.hsim() * z.hori();
  const int nborder = g.mirror ? z.nborder() : 0;
  float* sK = sm + (SIM ? 6 : 3) * n2;  // [hsim][hsim]
  float* sRK = sK + nsim;               // [hsim][hori] row sums
  float* sBK = sRK + nrow;              // mirror's border
  float* sS = sBK + nborder;            // SIM only: the same three maps of the similarity
  float* sRS = sS + nsim;
  float* sBS = sRS + nrow;
  const int tile = tile0 + blockIdx.x;
  const int ti = tile / g.ntx, tj = tile - ti * g.ntx;
  const int h0 = -g.ov + ti * g.step, w0 = -g.ov + tj * g.step;
  const int tid = threadIdx.x;
  // divergences from estimates that are all zero are zero (pixel_kl's r2 = 0)
  const bool kl_on = *nonzero != 0;
  for (int i = tid; i < n2; i += kThreads) {
    const int y = i / kTile, x = i - y * kTile;
    const size_t o = (size_t)clampn(h0 + y, 0, g.H - 1) * g.W + clampn(w0 + x, 0, g.W - 1);
    if (kl_on) {
      sRf[i] = rf[o];
      sPf[i] = pf[o];
      sCf[i] = cf[o];
    }
    if (SIM) {
      sA1[i] = a1[o];
      sA2[i] = a2[o];
      sDp[i] = dp[o];
    }
  }
  const int kc = z.wsh() * z.sws() + z.wsh();
  const size_t base = (size_t)blockIdx.x * z.sws() * z.sws() * npix;
  float* wt = wout + base;
  float* st = sums ? sums + base : nullptr;
  __syncthreads();
  // similarity and divergence of grid position i's pixel pair (c, q)
  auto evaluate = [&](int c, int q, float* s, float* k, int i) {
    if (SIM) s[i] = pixel_sim(sA1[c], sA2[c], sDp[c], sA1[q], sA2[q], sDp[q]);
    if (kl_on) k[i] = pixel_kl(sRf[c], sPf[c], sCf[c], sRf[q], sPf[q], sCf[q]);
  };
  // similarities and divergences of offset (hh, ww) on the whole grid, with
  // the two pixels swapped in the interior for the first wsh window rows (the
  // values the reference copies from the mirrored offset)
  auto direct = [&](int hh, int ww) {
    for (int it = tid; it < nsim; it += kThreads) {
      const int h = it / z.hsim(), w = it - h * z.hsim();
      const bool interior = h >= z.wsh() && w >= z.wsh() && w < z.hsim() - z.wsh();
      const int c = (h + z.wsh()) * kTile + (w + z.wsh()), q = (h + hh) * kTile + (w + ww);
      const bool swap = interior && hh < z.wsh();
      evaluate(swap ? q : c, swap ? c : q, sS, sK, it);
    }
  };
  // p-wide row sums of the maps; `at(h, w)` gives a map's value.  An item is
  // three adjacent sums from one load of their p + 2 values, each added left
  // to right.
  const int third = (z.hori() + 2) / 3;
  auto row_sums = [&](auto at) {
    for (int it = tid; it < z.hsim() * third; it += kThreads) {
      const int r = it / third, col = 3 * (it - r * third);
      float rs[3] = {0.0f, 0.0f, 0.0f}, rk[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int ky = 0; ky < z.p() + 2; ++ky) {
        if (col + ky >= z.hsim()) break;
        const float vs = SIM ? at(sS, sBS, r, col + ky) : 0.0f, vk = kl_on ? at(sK, sBK, r, col + ky) : 0.0f;
#pragma unroll
        for (int e = 0; e < 3; ++e)
          if (ky >= e && ky < z.p() + e) {
            if (SIM) rs[e] += vs;
            rk[e] += vk;
          }
      }
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (col + e < z.hori()) {
          if (SIM) sRS[r * z.hori() + col + e] = rs[e];
          if (kl_on) sRK[r * z.hori() + col + e] = rk[e];
        }
    }
  };
  auto direct_at = [&](const float* m, const float*, int h, int w) { return m[h * z.hsim() + w]; };
  // p-wide column sums and weights of offset k; an item is three rows of a
  // column, each sum added top down
  auto weights_of = [&](int k) {
    for (int it = tid; it < z.hori() * third; it += kThreads) {
      const int x3 = it / z.hori(), y = it - x3 * z.hori(), x = 3 * x3;
      float s[3], kl[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int kx = 0; kx < z.p() + 2; ++kx) {
        if (x + kx >= z.hsim()) break;
        const float vs = SIM ? sRS[(x + kx) * z.hori() + y] : 0.0f, vk = kl_on ? sRK[(x + kx) * z.hori() + y] : 0.0f;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          if (SIM && kx == e) s[e] = vs;
          if (SIM && kx > e && kx < z.p() + e) s[e] += vs;
          if (kx == e) kl[e] = vk;
          if (kx > e && kx < z.p() + e) kl[e] += vk;
        }
      }
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        if (x + e >= z.hori()) break;
        const size_t at = (size_t)k * npix + (x + e) * z.hori() + y;
        float t;
        if (SIM) {
          t = s[e] / g.h;
          if (st) st[at] = t;
        } else {
          t = st[at];
        }
        if (kl_on) t += kl[e] / g.T;
        float wv = expf(t);
        if (isnan(wv) || isinf(wv)) wv = 0.0f;
        if (k == kc) wv = 0.0f;
        wt[at] = wv;
      }
    }
  };
  const int u0 = nl_group(g, blockIdx.y, gridDim.y), u1 = nl_group(g, blockIdx.y + 1, gridDim.y);
  for (int u = u0; u < u1; ++u) {
    if (!g.mirror || u < z.sws()) {
      // an offset of the centre window row (or any one, without mirrors),
      // computed as the reference computes it
      const int hh = g.mirror ? z.wsh() : u / z.sws(), ww = g.mirror ? u : u - hh * z.sws();
      direct(hh, ww);
      __syncthreads();
      row_sums(direct_at);
      __syncthreads();
      weights_of(hh * z.sws() + ww);
      __syncthreads();
      continue;
    }
    // a lower-row offset with its mirror: the mirror's interior values are the
    // lower offset's maps shifted by the mirror's offset (the very values the
    // reference copies), its border values are computed here
    const int v = u - z.sws();
    const int hl = z.wsh() + 1 + v / z.sws(), wl = v % z.sws();
    const int hu = 2 * z.wsh() - hl, wu = 2 * z.wsh() - wl;
    const int top = z.wsh() * z.hsim(), band = 2 * z.wsh();
    for (int it = tid; it < nsim + nborder; it += kThreads) {
      if (it < nsim) {
        const int h = it / z.hsim(), w = it - h * z.hsim();
        evaluate((h + z.wsh()) * kTile + (w + z.wsh()), (h + hl) * kTile + (w + wl), sS, sK, it);
      } else {
        const int ib = it - nsim;
        int h, w;
        if (ib < top) {
          h = ib / z.hsim();
          w = ib - h * z.hsim();
        } else {
          const int j = ib - top;
          h = z.wsh() + j / band;
          const int m = j - (j / band) * band;
          w = m < z.wsh() ? m : z.hsim() - band + m;
        }
        evaluate((h + z.wsh()) * kTile + (w + z.wsh()), (h + hu) * kTile + (w + wu), sBS, sBK, ib);
      }
    }
    __syncthreads();
    row_sums(direct_at);
    __syncthreads();
    weights_of(hl * z.sws() + wl);
    __syncthreads();
    const int dh = hu - z.wsh(), dw = wu - z.wsh();
    row_sums([&](const float* m, const float* border, int h, int w) {
      if (h >= z.wsh() && w >= z.wsh() && w < z.hsim() - z.wsh()) return m[(h + dh) * z.hsim() + (w + dw)];
      return border[h < z.wsh() ? h * z.hsim() + w
                                : top + (h - z.wsh()) * band + (w < z.wsh() ? w : w - z.hsim() + band)];
    });
    __syncthreads();
    weights_of(hu * z.sws() + wu);
    __syncthreads();
  }
}

// whether any reflectivity estimate is not zero
__global__ void nlinsar_nonzero_kernel(const float* __restrict__ rf, size_t n, int* __restrict__ nonzero) {
  bool any = false;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    any = any || !(rf[i] == 0.0f);
  if (__syncthreads_or(any) && threadIdx.x == 0) *nonzero = 1;
}

// std::priority_queue<weight_el> of smoothing.cpp: a binary heap whose top is
// the smallest weight; push sifts up, pop moves the last element into the hole
// left by sifting the top down to a leaf and sifts it up again.
struct DevHeap {
  float w[kMaxLmin];
  int idx[kMaxLmin];
  int n = 0;
  __device__ static bool before(float aw, float bw) { return aw > bw; }
  __device__ void sift_up(int hole, float vw, int vi) {
    int parent = (hole - 1) / 2;
    while (hole > 0 && before(w[parent], vw)) {
      w[hole] = w[parent];
      idx[hole] = idx[parent];
      hole = parent;
      parent = (hole - 1) / 2;
    }
    w[hole] = vw;
    idx[hole] = vi;
  }
  __device__ void push(float vw, int vi) {
    ++n;
    sift_up(n - 1, vw, vi);
  }
  __device__ void pop() {
    const int len = n - 1;
    const float vw = w[len];
    const int vi = idx[len];
    int hole = 0, child = 0;
    while (child < (len - 1) / 2) {
      child = 2 * (child + 1);
      if (before(w[child], w[child - 1])) --child;
      w[hole] = w[child];
      idx[hole] = idx[child];
      hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
      child = 2 * (child + 1);
      w[hole] = w[child - 1];
      idx[hole] = idx[child - 1];
      hole = child - 1;
    }
    sift_up(hole, vw, vi);
    n = len;
  }
};

__global__ void __launch_bounds__(kEstThreads)
    nlinsar_estimate_kernel(const float* __restrict__ a1, const float* __restrict__ fa, const float* __restrict__ fr,
                            const float* __restrict__ fi, const float* __restrict__ prf,
                            const float* __restrict__ ppf, const float* __restrict__ pcf, float* __restrict__ orf,
                            float* __restrict__ opf, float* __restrict__ ocf, NlGeom g, int tile0,
                            const float* __restrict__ wts) {
  const int npix = g.hori * g.hori;
  const int pix = blockIdx.x * kEstThreads + threadIdx.x;
  if (pix >= npix) return;
  const int tile = tile0 + blockIdx.y;
  const int ti = tile / g.ntx, tj = tile - ti * g.ntx;
  const int h0 = -g.ov + ti * g.step, w0 = -g.ov + tj * g.step;
  const int x = pix / g.hori, y = pix - x * g.hori;
  // the output pixel this tile position writes last, if any
  const int ry = ti * g.step + x, rx = tj * g.step + y;  // = h0 + ov + x, w0 + ov + y
  int oy, ox;
  if (ry < g.H - 1) oy = ry;
  else if (ti == g.nty - 1 && x == g.hori - 1) oy = g.H - 1;
  else return;
  if (rx < g.W - 1) ox = rx;
  else if (tj == g.ntx - 1 && y == g.hori - 1) ox = g.W - 1;
  else return;
  const int no = g.sws * g.sws;
  const float* wp = wts + (size_t)blockIdx.y * no * npix + pix;
  // looks, the weights in the order of the weights kernel's units
  float s1 = 0.0f, s2 = 0.0f;
  auto look = [&](int k) {
    const float wv = wp[(size_t)k * npix];
    s1 += wv;
    s2 += wv * wv;
  };
  if (!g.mirror) {
#pragma unroll 4
    for (int k = 0; k < no; ++k) look(k);
  } else {
#pragma unroll 4
    for (int ww = 0; ww < g.sws; ++ww) look(g.wsh * g.sws + ww);
#pragma unroll 4
    for (int k = (g.wsh + 1) * g.sws; k < no; ++k) {
      look(k);
      look(no - 1 - k);  // the mirror
    }
  }
  // smoothing (smoothing.cpp:65-117)
  int sel[kMaxLmin];
  int nsel = 0;
  float wmean = 0.0f;
  if (s1 * s1 / s2 < (float)g.lmin) {
    DevHeap hp;
    const double as = a1[(size_t)clampn(h0 + x + g.ov, 0, g.H - 1) * g.W + clampn(w0 + y + g.ov, 0, g.W - 1)];
    for (int hh = 0; hh < g.sws; ++hh) {
      const int iy = clampn(h0 + x + g.ov + hh - g.wsh, 0, g.H - 1);
      for (int ww = 0; ww < g.sws; ++ww) {
        const float at = a1[(size_t)iy * g.W + clampn(w0 + y + g.ov + ww - g.wsh, 0, g.W - 1)];
        if (at < 2.0 * as) {
          const int k = hh * g.sws + ww;
          const float wk = wp[(size_t)k * npix];
          if (hp.n < g.lmin)
            hp.push(wk, k);
          else if (hp.w[0] < wk) {
            hp.pop();
            hp.push(wk, k);
          }
        }
      }
    }
    while (hp.n > 0) {
      wmean += hp.w[0];
      sel[nsel++] = hp.idx[0];
      hp.pop();
    }
    wmean /= (float)nsel;
    // ascending offsets for the merge below
    for (int i = 1; i < nsel; ++i) {
      const int v = sel[i];
      int j = i - 1;
      while (j >= 0 && sel[j] > v) {
        sel[j + 1] = sel[j];
        --j;
      }
      sel[j + 1] = v;
    }
  }
  // weighted means (compute_insar.cl:68-102)
  float N = 0.0f, A = 0.0f, Xr = 0.0f, Xi = 0.0f;
  int si = 0;
  for (int i = 0; i < g.sws; ++i) {
    const int iy = clampn(h0 + x + i + g.psh, 0, g.H - 1);
    for (int j = 0; j < g.sws; ++j) {
      const int k = i * g.sws + j;
      float wk = wp[(size_t)k * npix];
      if (si < nsel && sel[si] == k) {
        wk = wmean;
        ++si;
      }
      const size_t f = (size_t)iy * g.W + clampn(w0 + y + j + g.psh, 0, g.W - 1);
      N += wk;
      A += wk * fa[f];
      Xr += wk * fr[f];
      Xi += wk * fi[f];
    }
  }
  const float refl = A / N, phi = atan2f(Xi, Xr), coh = sqrtf(Xr * Xr + Xi * Xi) / A;
  const size_t o = (size_t)oy * g.W + ox;
  auto valid = [](float v) { return !(isnan(v) || isinf(v) || v == 0.0f); };
  orf[o] = valid(refl) ? refl : prf[o];
  if (valid(phi)) {
    float ph = phi;
    if (ph > 3.14159274101257324f) ph -= 2.0f * 3.14159274101257324f;
    if (ph < -3.14159274101257324f) ph += 2.0f * 3.14159274101257324f;
    opf[o] = ph;
  } else {
    opf[o] = ppf[o];
  }
  ocf[o] = valid(coh) ? fminf(1.0f, fmaxf(0.0f, coh)) : pcf[o];
}

size_t weights_smem(const NlGeom& g, bool sim) {
  const size_t maps = (size_t)g.hsim * g.hsim + (size_t)g.hsim * g.hori + (g.mirror ? (size_t)g.nborder : 0);
  return ((sim ? 6 : 3) * (size_t)kTile * kTile + (sim ? 2 : 1) * maps) * sizeof(float);
}

int nlinsar_geom(int H, int W, int sws, int p, int lmin, NlGeom& g) {
  if (H < 1 || W < 1) return set_error(DCL_ERR_INVALID_ARGUMENT, "height and width must be >= 1");
  if (sws < 1 || sws % 2 == 0 || p < 1 || p % 2 == 0)
    return set_error(DCL_ERR_INVALID_ARGUMENT, "search window and patch sizes must be odd");
  if (p != 3 && p != 7)
    return set_error(DCL_ERR_UNSUPPORTED,
                     "patch size %d: the reference's h is tabulated for 3 and 7 only (other sizes draw it from an "
                     "unseeded simulation, nlinsar.cpp:60-69)",
                     p);
  if (lmin < 1 || lmin > kMaxLmin) return set_error(DCL_ERR_UNSUPPORTED, "lmin must be in [1, %d]", kMaxLmin);
  g.H = H;
  g.W = W;
  g.sws = sws;
  g.wsh = (sws - 1) / 2;
  g.p = p;
  g.psh = (p - 1) / 2;
  g.ov = g.wsh + g.psh;
  g.hsim = kTile - sws + 1;
  g.hori = kTile - 2 * g.ov;
  // mirrored maps need an interior (rows from wsh, columns wsh .. hsim-wsh-1)
  // and room for the mirror's border values
  g.nborder = g.wsh * g.hsim + (g.hsim - g.wsh) * 2 * g.wsh;
  g.mirror = 2 * g.wsh < g.hsim ? 1 : 0;
  if (g.mirror && weights_smem(g, true) > 227 * 1024) g.mirror = 0;
  if (g.hori < 1) return set_error(DCL_ERR_UNSUPPORTED, "search window and patch too large for the 80 x 80 tiles");
  if (g.hori * g.hori > 6 * 1024 || weights_smem(g, true) > 227 * 1024)
    return set_error(DCL_ERR_UNSUPPORTED, "search window %d with patch %d: tile state exceeds shared memory", sws, p);
  g.step = kTile - 2 * g.ov;
  g.nty = 0;
  for (int h0 = -g.ov; h0 < H; h0 += g.step) ++g.nty;
  g.ntx = 0;
  for (int w0 = -g.ov; w0 < W; w0 += g.step) ++g.ntx;
  g.lmin = lmin;
  const int area = p * p;
  const float h_theo = p == 3 ? 0.58f : 0.244f;
  g.h = h_theo * area;
  g.T = (float)(2.0 / g.h * M_PI / 4 * area);
  return DCL_OK;
}

template <class Z, bool SIM>
cudaError_t launch_weights_t(const float* a1, const float* a2, const float* dp, float* const* est, const NlGeom& g,
                             int tile0, int tiles, int groups, const int* nonzero, float* sums, float* wts,
                             cudaStream_t st) {
  static size_t allowed[kMaxDevices];
  const size_t smem = weights_smem(g, SIM);
  const cudaError_t e = allow_dynamic_smem((const void*)nlinsar_weights_kernel<Z, SIM>, smem, allowed);
  if (e != cudaSuccess) return e;
  return launch_kernel(nlinsar_weights_kernel<Z, SIM>, dim3(tiles, groups), weights_threads(SIM), smem, st, a1, a2, dp,
                       est[0], est[1], est[2], g, tile0, nonzero, sums, wts);
}

template <bool SIM>
cudaError_t launch_weights(const float* a1, const float* a2, const float* dp, float* const* est, const NlGeom& g,
                           int tile0, int tiles, const int* nonzero, float* sums, float* wts, int sms,
                           cudaStream_t st) {
  // Groups of offsets per tile: waves of blocks (one or two per SM) times a block's
  // time, its share of a tile's work (about 4 ms) and staging (about 8 us).
  // One block per tile left 168 tiles of a 600 x 700 scene in two waves.
  int groups = 1;
  double best = 0.0;
  for (int z = 1; z <= std::min(64, nl_units(g)); ++z) {
    const int at_once = sms * (SIM ? 1 : 2);
    const double t = (double)(((long long)tiles * z + at_once - 1) / at_once) * (4000.0 / z + 8.0);
    if (best == 0.0 || t < best) {
      best = t;
      groups = z;
    }
  }
  auto go = [&](auto launch) { return launch(a1, a2, dp, est, g, tile0, tiles, groups, nonzero, sums, wts, st); };
  if (g.sws == 21 && g.p == 7) return go(launch_weights_t<NlSizes<21, 7>, SIM>);
  if (g.sws == 21 && g.p == 3) return go(launch_weights_t<NlSizes<21, 3>, SIM>);
  return go(launch_weights_t<NlSizes<0, 0>, SIM>);
}

}  // namespace

int nlinsar_check(int H, int W, int sws, int p, int lmin) {
  NlGeom g;
  return nlinsar_geom(H, W, sws, p, lmin, g);
}

// ref / phase / coh: initial estimates on entry, results on exit (device).
int nlinsar_device(const float* a1, const float* a2, const float* dp, float* ref, float* phase, float* coh, int H,
                   int W, int sws, int p, int niter, int lmin, cudaStream_t st) {
  if (!a1 || !a2 || !dp || !ref || !phase || !coh) return set_error(DCL_ERR_INVALID_ARGUMENT, "null pointer");
  if (niter < 0) return set_error(DCL_ERR_INVALID_ARGUMENT, "niter must be >= 0");
  int dev = 0;
  const int rc0 = ensure_device_ready(dev);
  if (rc0) return rc0;
  NlGeom g;
  int rc = nlinsar_geom(H, W, sws, p, lmin, g);
  if (rc) return rc;
  if (niter == 0) return DCL_OK;
  const size_t n = (size_t)H * W;
  const int ntiles = g.ntx * g.nty;
  const size_t npix = (size_t)g.hori * g.hori, no = (size_t)sws * sws;
  const size_t per_tile = no * npix * sizeof(float);
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>(ntiles, kWeightsBytes / per_tile));
  // the first pass's patch sums of the similarities, where the later passes
  // can keep them (a second scratch of at most the weights' size)
  const size_t sum_bytes = niter > 1 && chunk == ntiles ? (size_t)ntiles * per_tile : 0;
  char* buf = nullptr;
  const size_t fixed = 6 * n * sizeof(float) + 256 + (size_t)chunk * per_tile;
  cudaError_t e = cudaMallocAsync(&buf, fixed + sum_bytes, st);
  bool keep = sum_bytes > 0;
  if (e == cudaErrorMemoryAllocation && keep) {
    cudaGetLastError();
    keep = false;
    e = cudaMallocAsync(&buf, fixed, st);
  }
  if (e != cudaSuccess) return cuda_error(e, "cudaMallocAsync(NL-InSAR)");
  int* nonzero = reinterpret_cast<int*>(buf);
  float* fa = reinterpret_cast<float*>(buf + 256);
  float *fr = fa + n, *fi = fr + n, *tr = fi + n, *tp = tr + n, *tc = tp + n;
  float* wts = tc + n;
  float* sums = keep ? wts + (size_t)chunk * no * npix : nullptr;
  e = cudaMemsetAsync(nonzero, 0, sizeof(int), st);
  if (e == cudaSuccess) {
    const int sms = sm_count(dev);
    e = launch_kernel(nlinsar_filter_values_kernel, (unsigned)((n + 255) / 256), 256, 0, st, a1, a2, dp, fa, fr, fi, n);
    profile_count(1);
    // estimates ping-pong between the caller's planes and tr/tp/tc; an odd
    // number of passes ends in tr/tp/tc and is copied back
    float* cur[3] = {ref, phase, coh};
    float* nxt[3] = {tr, tp, tc};
    for (int it = 0; it < niter && e == cudaSuccess; ++it) {
      e = launch_kernel(nlinsar_nonzero_kernel, (unsigned)std::min<size_t>((n + 1023) / 1024, 8 * sms), 256, 0, st,
                        cur[0], n, nonzero);
      for (int t0 = 0; t0 < ntiles && e == cudaSuccess; t0 += chunk) {
        const int nt = std::min(chunk, ntiles - t0);
        e = keep && it > 0 ? launch_weights<false>(a1, a2, dp, cur, g, t0, nt, nonzero, sums, wts, sms, st)
                           : launch_weights<true>(a1, a2, dp, cur, g, t0, nt, nonzero, sums, wts, sms, st);
        const dim3 grid((unsigned)((npix + kEstThreads - 1) / kEstThreads), nt);
        if (e == cudaSuccess)
          e = launch_kernel(nlinsar_estimate_kernel, grid, kEstThreads, 0, st, a1, fa, fr, fi, cur[0], cur[1], cur[2],
                            nxt[0], nxt[1], nxt[2], g, t0, wts);
        profile_count(2);
      }
      profile_count(1);
      std::swap(cur, nxt);
    }
    if (cur[0] != ref)
      for (int d = 0; d < 3 && e == cudaSuccess; ++d)
        e = cudaMemcpyAsync(d == 0 ? ref : (d == 1 ? phase : coh), cur[d], n * sizeof(float),
                            cudaMemcpyDeviceToDevice, st);
  }
  cudaFreeAsync(buf, st);
  if (e != cudaSuccess) return cuda_error(e, "NL-InSAR");
  return DCL_OK;
}

}  // namespace dcl

extern "C" int dcl_nlinsar_device(const float* a1, const float* a2, const float* phi, float* ref, float* phase,
                                  float* coh, int H, int W, int search_window_size, int patch_size, int niter, int lmin,
                                  void* stream) {
  return dcl::nlinsar_device(a1, a2, phi, ref, phase, coh, H, W, search_window_size, patch_size, niter, lmin,
                             (cudaStream_t)stream);
}

extern "C" int dcl_nlinsar(const float* a1, const float* a2, const float* phi, float* ref, float* phase, float* coh,
                           int H, int W, int search_window_size, int patch_size, int niter, int lmin) {
  if (!a1 || !a2 || !phi || !ref || !phase || !coh) return dcl::set_error(DCL_ERR_INVALID_ARGUMENT, "null pointer");
  const int vr = dcl::nlinsar_check(H, W, search_window_size, patch_size, lmin);
  if (vr) return vr;
  if (niter < 0) return dcl::set_error(DCL_ERR_INVALID_ARGUMENT, "niter must be >= 0");
  cudaStream_t st = cudaStreamPerThread;
  const size_t n = (size_t)H * W, b = n * sizeof(float);
  float* buf = nullptr;
  cudaError_t e = cudaMallocAsync(&buf, 6 * b, st);
  if (e != cudaSuccess) return dcl::cuda_error(e, "cudaMallocAsync(NL-InSAR)");
  const float* hin[6] = {a1, a2, phi, ref, phase, coh};
  for (int d = 0; d < 6 && e == cudaSuccess; ++d)
    e = cudaMemcpyAsync(buf + d * n, hin[d], b, cudaMemcpyHostToDevice, st);
  int rc = DCL_OK;
  if (e != cudaSuccess) rc = dcl::cuda_error(e, "cudaMemcpyAsync(H2D)");
  if (rc == DCL_OK)
    rc = dcl::nlinsar_device(buf, buf + n, buf + 2 * n, buf + 3 * n, buf + 4 * n, buf + 5 * n, H, W,
                             search_window_size, patch_size, niter, lmin, st);
  if (rc == DCL_OK) {
    float* hout[3] = {ref, phase, coh};
    for (int d = 0; d < 3 && e == cudaSuccess; ++d)
      e = cudaMemcpyAsync(hout[d], buf + (3 + d) * n, b, cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) rc = dcl::cuda_error(e, "cudaMemcpyAsync(D2H)");
  }
  cudaFreeAsync(buf, st);
  e = cudaStreamSynchronize(st);
  if (rc == DCL_OK && e != cudaSuccess) rc = dcl::cuda_error(e, "NL-InSAR");
  return rc;
}

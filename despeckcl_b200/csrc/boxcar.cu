// Boxcar InSAR filter: w x w window means of the intensity and of the complex
// interferogram (src/compute/boxcar/cl_kernels/boxcar_kernel.cl:19-69 in the
// reference, driven by src/compute/boxcar/boxcar.cpp:30-100 over 512x512 tiles
// with overlap (w-1)/2).
//
// One pass over HBM: each CTA stages its output tile plus a (w-1)/2 halo of
// (I, Re, Im) = ((a1^2+a2^2)/2, a1 a2 cos phi, a1 a2 sin phi) in shared memory,
// forms horizontal window sums, then vertical sums, and writes
// ref = mean I, phase = atan2(Im, Re), coh = |sum Re + j Im| / sum I.  On large
// scenes with windows up to 7 x 7 warps walk down the scene instead, the sums
// in registers (boxcar_walk_kernel).
//
// Like NL-SAR, the reference's clamped tile write-back puts the result of
// virtual row H-1+(w-1)/2 of the clamp-extended image into output row H-1
// (and likewise for the last column); the kernel computes on that virtual
// plane.

#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/despeckcl_b200.h"
#include "dcl_internal.h"
#include "fast_math.cuh"

namespace dcl {
namespace {

constexpr int kBoxTW = 64;
constexpr int kBoxTH = 32;  // 40- and 48-row tiles (2 CTAs per SM) measured slower
constexpr int kBoxThreads = kBoxTH * 8;  // one vertical item (4 rows x 2 columns) per thread
constexpr int kBoxMaxR = 15;

__device__ __forceinline__ int clampi_b(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__global__ void __launch_bounds__(kBoxThreads)
    boxcar_kernel(const float* __restrict__ a1, const float* __restrict__ a2, const float* __restrict__ phi,
                  float* __restrict__ ref, float* __restrict__ phase, float* __restrict__ coh, int H, int W, int r) {
  extern __shared__ float sm[];
  const int SW = kBoxTW + 2 * r, SH = kBoxTH + 2 * r;
  float* sI = sm;                 // [SH][SW]
  float* sR = sI + SH * SW;
  float* sJ = sR + SH * SW;
  float* hI = sJ + SH * SW;       // [SH][kBoxTW] horizontal sums
  float* hR = hI + SH * kBoxTW;
  float* hJ = hR + SH * kBoxTW;
  const int vy0 = blockIdx.y * kBoxTH, vx0 = blockIdx.x * kBoxTW;
  const int tid = threadIdx.x;
  for (int i = tid; i < SH * SW; i += kBoxThreads) {
    const int rr = i / SW, cc = i - rr * SW;
    const int y = clampi_b(vy0 - r + rr, 0, H - 1), x = clampi_b(vx0 - r + cc, 0, W - 1);
    const size_t g = (size_t)y * W + x;
    const float am = a1[g], as = a2[g];
    float sn, cs;
    __sincosf(phi[g], &sn, &cs);
    const float aa = am * as;
    sI[i] = (am * am + as * as) / 2;
    sR[i] = aa * cs;
    sJ[i] = aa * sn;
  }
  __syncthreads();
  for (int i = tid; i < SH * kBoxTW; i += kBoxThreads) {
    const int rr = i / kBoxTW, cc = i - rr * kBoxTW;
    const float* pI = sI + rr * SW + cc;
    const float* pR = sR + rr * SW + cc;
    const float* pJ = sJ + rr * SW + cc;
    float si = 0.f, sr = 0.f, sj = 0.f;
    for (int k = 0; k <= 2 * r; ++k) {
      si += pI[k];
      sr += pR[k];
      sj += pJ[k];
    }
    hI[i] = si;
    hR[i] = sr;
    hJ[i] = sj;
  }
  __syncthreads();
  const float inv_n = 1.0f / (float)((2 * r + 1) * (2 * r + 1));
  for (int i = tid; i < kBoxTH * kBoxTW; i += kBoxThreads) {
    const int rr = i / kBoxTW, cc = i - rr * kBoxTW;
    const int vy = vy0 + rr, vx = vx0 + cc;
    const int oy = (vy < H - 1) ? vy : (vy == H - 1 + r ? H - 1 : -1);
    const int ox = (vx < W - 1) ? vx : (vx == W - 1 + r ? W - 1 : -1);
    if (oy < 0 || ox < 0) continue;
    float si = 0.f, sr = 0.f, sj = 0.f;
    for (int k = 0; k <= 2 * r; ++k) {
      si += hI[(rr + k) * kBoxTW + cc];
      sr += hR[(rr + k) * kBoxTW + cc];
      sj += hJ[(rr + k) * kBoxTW + cc];
    }
    const size_t o = (size_t)oy * W + ox;
    ref[o] = si * inv_n;
    phase[o] = atan2_fast(sj, sr);
    coh[o] = sqrtf(sr * sr + sj * sj) / si;
  }
}

// |sum| / sum I from 2 I sums, with the hardware square root and the fast
// division (a few ulps, against the 1e-4 relative tolerance of the coherence)
__device__ __forceinline__ float boxcar_coherence(float sr, float sj, float si) {
  float m;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(m) : "f"(__fmaf_rn(sr, sr, __fmul_rn(sj, sj))));
  return __fdividef(2.0f * m, si);
}

// Packed and scalar adds for the window sums: (Re, Im) pairs are summed two
// lanes at a time with the f32x2 add (each component rounded like a scalar
// add).
__device__ __forceinline__ float wadd(float a, float b) { return a + b; }
__device__ __forceinline__ float2 wadd(float2 a, float2 b) { return __fadd2_rn(a, b); }

// Window sums of 4 consecutive outputs o[q] = v[q] + ... + v[q + w - 1],
// q = 0..3, from the 4 + w - 1 values v: the part v[3 .. w-1] that all four
// windows share is added once, then each window adds its own ends (w + 6 adds
// instead of 4 w).  No term is subtracted, so no sum cancels.
template <int R, class T>
__device__ __forceinline__ void window4(const T* v, T* o) {
  constexpr int w = 2 * R + 1;
  if (w < 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      T acc = v[q];
#pragma unroll
      for (int k = 1; k < w; ++k) acc = wadd(acc, v[q + k]);
      o[q] = acc;
    }
    return;
  }
  T c = v[3];
#pragma unroll
  for (int k = 4; k < w; ++k) c = wadd(c, v[k]);
  const T l1 = wadd(v[1], v[2]);
  const T l0 = wadd(v[0], l1);
  const T r2 = wadd(v[w], v[w + 1]);
  const T r3 = wadd(r2, v[w + 2]);
  o[0] = wadd(l0, c);
  o[1] = wadd(wadd(l1, c), v[w]);
  o[2] = wadd(wadd(v[2], c), r2);
  o[3] = wadd(c, r3);
}

// Window sums of 2 consecutive outputs from the w + 1 values v: the middle
// v[1 .. w-1] is summed once (w + 1 adds instead of 2 (w - 1)).
template <int R, class T>
__device__ __forceinline__ void window2(const T* v, T& o0, T& o1) {
  constexpr int w = 2 * R + 1;
  if (w == 1) {
    o0 = v[0];
    o1 = v[1];
    return;
  }
  T m = v[1];
#pragma unroll
  for (int k = 2; k < w; ++k) m = wadd(m, v[k]);
  o0 = wadd(v[0], m);
  o1 = wadd(m, v[w]);
}

// Compile-time window radius R (w = 2R+1 <= 15): a 64 x 32 tile per CTA of
// 256 threads.  The staged tile holds the intensity I as one plane and the
// interferogram (Re, Im) as interleaved pairs, so both complex window sums
// run as packed f32x2 adds:
//   horizontal pass: window4 over one row x 4 columns of I and window2 over
//     one row x 2 columns of (Re, Im), from 16-byte loads;
//   vertical pass, 4 rows x 2 columns per thread (the 256 items of a tile):
//     window4 down the column pair of I and down each column's (Re, Im),
//     all as packed adds, from 8- and 16-byte loads;
//   output: ref = mean I, phase = atan2(Im, Re), coh = |sum| / sum I, written
//     as 8-byte vectors where both columns are interior and the planes allow
//     it.
template <int R>
__global__ void __launch_bounds__(kBoxThreads)
    boxcar_r_kernel(const float* __restrict__ a1, const float* __restrict__ a2, const float* __restrict__ phi,
                    float* __restrict__ ref, float* __restrict__ phase, float* __restrict__ coh, int H, int W,
                    int vec_out) {
  // staged rows of SW values, pitch SWP (a multiple of 4: the horizontal
  // pass reads its windows as aligned 16-byte vectors, conflict free)
  constexpr int SW = kBoxTW + 2 * R, SH = kBoxTH + 2 * R, N = 4 + 2 * R;
  constexpr int SWP = (SW + 3) / 4 * 4, NQ = (N + 3) / 4;
  constexpr int HG = kBoxTW / 4;
  static_assert(4 * (HG - 1) + 4 * NQ <= SWP && (kBoxTW - 2) + 2 * (R + 1) <= SWP,
                "window vectors stay inside a staged row");
  static_assert((kBoxTH / 4) * (kBoxTW / 2) == kBoxThreads, "one vertical item per thread");
  extern __shared__ __align__(16) float sm[];
  float* sI = sm;                                              // [SH][SWP]: 2 I = a1^2 + a2^2
  float2* sZ = reinterpret_cast<float2*>(sm + SH * SWP);        // [SH][SWP] (Re, Im)
  float* hI = sm + 3 * SH * SWP;                               // [SH][kBoxTW] horizontal sums
  float2* hZ = reinterpret_cast<float2*>(hI + SH * kBoxTW);     // [SH][kBoxTW]
  const int vy0 = blockIdx.y * kBoxTH, vx0 = blockIdx.x * kBoxTW;
  const int tid = threadIdx.x;
  // staging: each thread issues the loads of U pixels (all of its share, up
  // to 12) before using any of them, so up to 3U loads per thread are in
  // flight (the staging is bound by memory latency, not bandwidth, at one
  // load in flight per plane).  A thread's staged pixels are i = tid + u T
  // (T threads); their (row, column) advance by (T / SW, T % SW) with one
  // carry, with no division.  Tiles whose staged region lies inside the
  // scene (all but the edge tiles) read without clamping, at 32-bit offsets
  // from the tile's first staged pixel.
  constexpr int U = (SH * SW + kBoxThreads - 1) / kBoxThreads < 12 ? (SH * SW + kBoxThreads - 1) / kBoxThreads : 12;
  constexpr int DR = (U * kBoxThreads) / SW, DC = (U * kBoxThreads) % SW;
  constexpr int dr = kBoxThreads / SW, dc = kBoxThreads % SW;
  const bool interior = vy0 >= R && vy0 + kBoxTH + R <= H && vx0 >= R && vx0 + kBoxTW + R <= W;
  const size_t base = interior ? (size_t)(vy0 - R) * W + (vx0 - R) : 0;
  const float* b1 = a1 + base;
  const float* b2 = a2 + base;
  const float* bp = phi + base;
  int rr0 = tid / SW, cc0 = tid - (tid / SW) * SW;
  for (int i0 = tid; i0 < SH * SW; i0 += U * kBoxThreads) {
    float am[U], as[U], ph[U];
    int sidx[U];
    {
      int rr = rr0, cc = cc0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kBoxThreads;
        if (i < SH * SW) {
          int off;
          if (interior) {
            off = rr * W + cc;
          } else {
            const int y = clampi_b(vy0 - R + rr, 0, H - 1), x = clampi_b(vx0 - R + cc, 0, W - 1);
            off = 0;
            am[u] = __ldg(a1 + (size_t)y * W + x);
            as[u] = __ldg(a2 + (size_t)y * W + x);
            ph[u] = __ldg(phi + (size_t)y * W + x);
          }
          if (interior) {
            am[u] = __ldg(b1 + off);
            as[u] = __ldg(b2 + off);
            ph[u] = __ldg(bp + off);
          }
          sidx[u] = rr * SWP + cc;
        }
        rr += dr;
        cc += dc;
        if (cc >= SW) {
          cc -= SW;
          ++rr;
        }
      }
    }
    rr0 += DR;
    cc0 += DC;
    if (cc0 >= SW) {
      cc0 -= SW;
      ++rr0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kBoxThreads;
      if (i < SH * SW) {
        const int si = sidx[u];
        float sn, cs;
        __sincosf(ph[u], &sn, &cs);
        const float aa = am[u] * as[u];
        // twice the intensity (I1 + I2): the halving is folded into the
        // output stage (exact: a power of two)
        sI[si] = am[u] * am[u] + as[u] * as[u];
        sZ[si] = make_float2(aa * cs, aa * sn);
      }
    }
  }
  __syncthreads();
  // horizontal: items of I (row, 4 columns: window4 from 16-byte loads) and
  // of (Re, Im) (row, 2 columns: window2 from 16-byte loads of 2 pairs);
  // consecutive lanes read consecutive 16-byte vectors of one row
  constexpr int NI = SH * HG, NZ = SH * (kBoxTW / 2);
  for (int it = tid; it < NI + NZ; it += kBoxThreads) {
    if (it < NI) {
      const int rr = it / HG, c0 = (it - rr * HG) * 4;
      const float4* src = reinterpret_cast<const float4*>(sI + rr * SWP + c0);
      float v[4 * NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const float4 t = src[q];
        v[4 * q] = t.x;
        v[4 * q + 1] = t.y;
        v[4 * q + 2] = t.z;
        v[4 * q + 3] = t.w;
      }
      float o[4];
      window4<R>(v, o);
      *reinterpret_cast<float4*>(hI + rr * kBoxTW + c0) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
      const int j = it - NI;
      const int rr = j / (kBoxTW / 2), c0 = (j - rr * (kBoxTW / 2)) * 2;
      const float4* src = reinterpret_cast<const float4*>(sZ + rr * SWP + c0);
      float2 v[2 + 2 * R + 1];
#pragma unroll
      for (int q = 0; q < R + 1; ++q) {
        const float4 t = src[q];
        v[2 * q] = make_float2(t.x, t.y);
        v[2 * q + 1] = make_float2(t.z, t.w);
      }
      float2 o0, o1;
      window2<R>(v, o0, o1);
      *reinterpret_cast<float4*>(hZ + rr * kBoxTW + c0) = make_float4(o0.x, o0.y, o1.x, o1.y);
    }
  }
  __syncthreads();
  // vertical: this thread's 4 rows x 2 columns (a warp covers 4 rows of the
  // tile's 64 columns): window4 down the column pair of I and down each
  // column's (Re, Im), all as packed adds
  const int c0 = (tid % (kBoxTW / 2)) * 2, r0 = (tid / (kBoxTW / 2)) * 4;
  float2 sIp[4];     // [row]: (I of column c0, I of column c0 + 1)
  float2 sZc[2][4];  // [column][row]: (Re, Im)
  {
    float2 vi[N], vz0[N], vz1[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      vi[k] = *reinterpret_cast<const float2*>(hI + (r0 + k) * kBoxTW + c0);
      const float4 t = *reinterpret_cast<const float4*>(hZ + (r0 + k) * kBoxTW + c0);
      vz0[k] = make_float2(t.x, t.y);
      vz1[k] = make_float2(t.z, t.w);
    }
    window4<R>(vi, sIp);
    window4<R>(vz0, sZc[0]);
    window4<R>(vz1, sZc[1]);
  }
  // outputs on the virtual plane: row H-1 holds virtual row H-1+R (likewise
  // column W-1); a column pair wholly left of column W-1 maps to itself
  // the staged plane holds 2 I: ref = (2 I sum) / (2 n), coh = 2 |sum| / (2 I sum)
  const float inv_2n = 0.5f / (float)((2 * R + 1) * (2 * R + 1));
  const int vx = vx0 + c0;
  const bool cols_plain = vx + 1 < W - 1;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int vy = vy0 + r0 + q;
    const int oy = (vy < H - 1) ? vy : (vy == H - 1 + R ? H - 1 : -1);
    if (oy < 0) continue;
    float o_r[2], o_p[2], o_c[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float si = e == 0 ? sIp[q].x : sIp[q].y;
      const float sr = sZc[e][q].x, sj = sZc[e][q].y;
      o_r[e] = si * inv_2n;
      o_p[e] = atan2_fast(sj, sr);
      o_c[e] = boxcar_coherence(sr, sj, si);
    }
    const size_t rowo = (size_t)oy * W;
    if (cols_plain && vec_out) {
      *reinterpret_cast<float2*>(ref + rowo + vx) = make_float2(o_r[0], o_r[1]);
      *reinterpret_cast<float2*>(phase + rowo + vx) = make_float2(o_p[0], o_p[1]);
      *reinterpret_cast<float2*>(coh + rowo + vx) = make_float2(o_c[0], o_c[1]);
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int x = vx + e;
        const int ox = (x < W - 1) ? x : (x == W - 1 + R ? W - 1 : -1);
        if (ox < 0) continue;
        ref[rowo + ox] = o_r[e];
        phase[rowo + ox] = o_p[e];
        coh[rowo + ox] = o_c[e];
      }
    }
  }
}

// Window radius 1 <= R <= 3 on large scenes: a warp walks down a strip of 128
// columns, each lane owning four adjacent ones.  The pixels of a row come by
// asynchronous copies, one 16-byte vector per lane and plane, into the warp's
// ring in shared memory a few rows ahead; the R columns on either side come
// from the neighbour lanes by shuffles (the strip's outer lanes only supply
// them); the horizontal sums of the last 2 R rows stay in registers, and each
// row of windows is written as soon as its last row has come in.  The sums are
// those of boxcar_r_kernel in the same order (its items are four columns of I,
// two of (Re, Im) and four rows, from the same origins), so the results are
// the same bits.
//
// VEC: all planes and rows are 16-byte aligned.  Otherwise, and at the scene's
// edges, the copies are single values, 32 adjacent columns at a time, and the
// results reach memory the same way through shared memory.
//
// 8192 x 8192, 7 x 7: the tiled kernel takes 425 us, bound by shared memory
// (79 %) and issue (137 thread instructions per pixel); this one takes
// 312 us (5.1 TB/s of the six planes) at 98 instructions per pixel (among other
// work 441 and 354 us).  Registers
// set its pace: 158 of them and twelve warps per SM.  Held to 128 for sixteen
// warps it spills and takes 530 us or more; with all rows of a group summed
// before the first output it needs 218 and takes 425 us.  A ring of eight rows
// takes 330 us, walks of 128 rows 334 us, of 32 rows 325 us.
constexpr int kWalkWarps = 4;
constexpr int kWalkCols = 120;  // columns a warp outputs
constexpr int kWalkRing = 4;   // rows in flight per warp
constexpr int kWalkBlocks = 3;  // per SM
constexpr int kWalkGroups = 16;  // groups of four rows a warp outputs at most

template <int R, bool VEC>
__global__ void __launch_bounds__(32 * kWalkWarps, kWalkBlocks)
    boxcar_walk_kernel(const float* __restrict__ a1, const float* __restrict__ a2, const float* __restrict__ phi,
                       float* __restrict__ ref, float* __restrict__ phase, float* __restrict__ coh, int H, int W,
                       int groups) {
  static_assert(R >= 1 && R <= 3, "registers; the halo comes from one neighbour lane");
  constexpr int w = 2 * R + 1;
  const int lane = threadIdx.x & 31;
  const int xs = (int)(blockIdx.x * kWalkWarps + (threadIdx.x >> 5)) * kWalkCols - 4;  // the strip's first column
  const int x0 = xs + 4 * lane;
  const int vW = W - 1 + R, vH = H - 1 + R;
  if (xs + 4 > vW) return;  // whole warp
  const int y0 = (int)blockIdx.y * groups * 4;
  const bool inside = xs >= 0 && xs + 128 <= W;
  const bool plain = xs + 124 < W;  // all output columns map to themselves
  const bool writes = lane >= 1 && lane <= 30;
  const float inv_2n = 0.5f / (float)(w * w);

  __shared__ __align__(16) float ring_s[kWalkWarps][kWalkRing][3][128];
  __shared__ __align__(16) float out_s[VEC ? 1 : kWalkWarps][3][128];
  float(*ring)[3][128] = ring_s[threadIdx.x >> 5];
  int slot = 0;
  int y = y0 - R;  // of the row to fetch next
  auto fetch = [&] {
    const size_t row = (size_t)clampi_b(y, 0, H - 1) * W;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const float* src = (p == 0 ? a1 : p == 1 ? a2 : phi) + row;
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(&ring[slot][p][0]);
      if (VEC && inside) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * lane), "l"(src + x0) : "memory");
      } else if (inside) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * lane + 128 * k),
                       "l"(src + xs + lane + 32 * k)
                       : "memory");
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * lane + 128 * k),
                       "l"(src + clampi_b(xs + lane + 32 * k, 0, W - 1))
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ++y;
    slot = slot + 1 == kWalkRing ? 0 : slot + 1;
  };
  struct Row {
    float2 I[2];  // horizontal sums of 2 I, columns in pairs
    float2 Z[4];  // and of (Re, Im)
  };
  // the horizontal sums of the next row, whose place takes the row kWalkRing
  // further
  auto next_row = [&](Row& h) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kWalkRing - 1) : "memory");
    __syncwarp();  // every lane's copies
    const float4 m4 = reinterpret_cast<const float4*>(ring[slot][0])[lane],
                 s4 = reinterpret_cast<const float4*>(ring[slot][1])[lane],
                 p4 = reinterpret_cast<const float4*>(ring[slot][2])[lane];
    const float am[4] = {m4.x, m4.y, m4.z, m4.w};
    const float as[4] = {s4.x, s4.y, s4.z, s4.w};
    const float ph[4] = {p4.x, p4.y, p4.z, p4.w};
    float v[4 + 2 * R];
    float2 z[4 + 2 * R];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float sn, cs;
      __sincosf(ph[c], &sn, &cs);
      const float aa = am[c] * as[c];
      // twice the intensity: the halving is folded into the output
      v[R + c] = am[c] * am[c] + as[c] * as[c];
      z[R + c] = make_float2(aa * cs, aa * sn);
    }
    __syncwarp();  // the row is read
    fetch();
#pragma unroll
    for (int b = 1; b <= R; ++b) {
      v[R - b] = __shfl_up_sync(0xffffffffu, v[R + 4 - b], 1);
      v[R + 3 + b] = __shfl_down_sync(0xffffffffu, v[R + b - 1], 1);
      z[R - b].x = __shfl_up_sync(0xffffffffu, z[R + 4 - b].x, 1);
      z[R - b].y = __shfl_up_sync(0xffffffffu, z[R + 4 - b].y, 1);
      z[R + 3 + b].x = __shfl_down_sync(0xffffffffu, z[R + b - 1].x, 1);
      z[R + 3 + b].y = __shfl_down_sync(0xffffffffu, z[R + b - 1].y, 1);
    }
    float o[4];
    window4<R>(v, o);
    h.I[0] = make_float2(o[0], o[1]);
    h.I[1] = make_float2(o[2], o[3]);
    window2<R>(z, h.Z[0], h.Z[1]);
    window2<R>(z + 2, h.Z[2], h.Z[3]);
  };
  auto add = [](const Row& a, const Row& b) {
    Row r;
#pragma unroll
    for (int c = 0; c < 2; ++c) r.I[c] = wadd(a.I[c], b.I[c]);
#pragma unroll
    for (int c = 0; c < 4; ++c) r.Z[c] = wadd(a.Z[c], b.Z[c]);
    return r;
  };
  auto write = [&](const Row& s, int vy) {
    const int oy = (vy < H - 1) ? vy : (vy == vH ? H - 1 : -1);
    if (oy < 0) return;
    float o_r[4], o_p[4], o_c[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float si = c & 1 ? s.I[c / 2].y : s.I[c / 2].x;
      o_r[c] = si * inv_2n;
      o_p[c] = atan2_fast(s.Z[c].y, s.Z[c].x);
      o_c[c] = boxcar_coherence(s.Z[c].x, s.Z[c].y, si);
    }
    const size_t rowo = (size_t)oy * W;
    if (VEC && plain) {
      if (!writes) return;
      *reinterpret_cast<float4*>(ref + rowo + x0) = make_float4(o_r[0], o_r[1], o_r[2], o_r[3]);
      *reinterpret_cast<float4*>(phase + rowo + x0) = make_float4(o_p[0], o_p[1], o_p[2], o_p[3]);
      *reinterpret_cast<float4*>(coh + rowo + x0) = make_float4(o_c[0], o_c[1], o_c[2], o_c[3]);
      return;
    }
    if (!VEC && plain) {
      // rows of any alignment: through shared memory, so that a store covers
      // 32 adjacent columns
      float(*o)[128] = out_s[threadIdx.x >> 5];
      __syncwarp();  // the row before is written
      reinterpret_cast<float4*>(o[0])[lane] = make_float4(o_r[0], o_r[1], o_r[2], o_r[3]);
      reinterpret_cast<float4*>(o[1])[lane] = make_float4(o_p[0], o_p[1], o_p[2], o_p[3]);
      reinterpret_cast<float4*>(o[2])[lane] = make_float4(o_c[0], o_c[1], o_c[2], o_c[3]);
      __syncwarp();
      const size_t at = rowo + xs + 4 + lane;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k == 3 && lane >= kWalkCols - 96) break;
        ref[at + 32 * k] = o[0][4 + lane + 32 * k];
        phase[at + 32 * k] = o[1][4 + lane + 32 * k];
        coh[at + 32 * k] = o[2][4 + lane + 32 * k];
      }
      return;
    }
    if (!writes) return;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int x = x0 + c;
      const int ox = (x < W - 1) ? x : (x == vW ? W - 1 : -1);
      if (ox < 0) continue;
      ref[rowo + ox] = o_r[c];
      phase[rowo + ox] = o_p[c];
      coh[rowo + ox] = o_c[c];
    }
  };

#pragma unroll
  for (int b = 0; b < kWalkRing; ++b) fetch();
  Row v[2 * R + 4];  // rows of a group of four windows; the first 2 R stay for the next
#pragma unroll
  for (int b = 0; b < 2 * R; ++b) next_row(v[b]);
  for (int g = 0; g < groups; ++g) {
    const int vy = y0 + 4 * g;
    if (vy > vH) break;
    // window4's sums, each output as soon as its last row is there
    if (R == 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        next_row(v[q + 2]);
        write(add(add(v[q], v[q + 1]), v[q + 2]), vy + q);
      }
    } else {
      next_row(v[w - 1]);
      Row c = v[3];
#pragma unroll
      for (int k = 4; k < w; ++k) c = add(c, v[k]);
      const Row l1 = add(v[1], v[2]);
      write(add(add(v[0], l1), c), vy);
      const Row t1 = add(l1, c), t2 = add(v[2], c);
      next_row(v[w]);
      write(add(t1, v[w]), vy + 1);
      next_row(v[w + 1]);
      const Row r2 = add(v[w], v[w + 1]);
      write(add(t2, r2), vy + 2);
      next_row(v[w + 2]);
      write(add(c, add(r2, v[w + 2])), vy + 3);
    }
#pragma unroll
    for (int b = 0; b < 2 * R; ++b) v[b] = v[b + 4];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

int walk_strips(int W, int R) { return (W - 1 + R) / kWalkCols + 1; }
int walk_blocks_x(int W, int R) { return (walk_strips(W, R) + kWalkWarps - 1) / kWalkWarps; }

// Whether the walk takes a scene: it wins once the scene gives every SM its
// twelve warps (3 x 3 and 7 x 7 take 41 and 47 us at 2500 x 2503, tiled 49 and
// 50; 31 and 38 at 2100 x 2203, 36 and 37; 12.4 and 14.5 at 1024 x 1024, 9.6
// and 10.8) and its strips fit the width.  A row costs its strips, half a strip
// for each idle warp of its last block, about half for the scalar copies of the
// outer strips, and 3.5 more where the last strip has next to no columns (it
// then holds up its block); the width's share of that has to reach a line that
// depends on the window and on the copies.  Measured with windows 3, 5 and 7 at
// 5 to 40 Mpx and 40 widths from 40 to 8192: below the lines the walk takes up
// to 4.4 times the tiles' time (40 wide), 1.6 (481), 1.37 (1200, 7 x 7), and
// down to 0.8 (960, 3 x 3); above them 0.65 to 1.02 of it.
bool walk_pays(int H, int W, int R, bool vec) {
  if ((long long)H * W < 5LL << 20) return false;
  const int strips = walk_strips(W, R), idle = walk_blocks_x(W, R) * kWalkWarps - strips;
  const int last = W + R - (strips - 1) * kWalkCols;  // columns of the last strip
  const double full = (double)W / kWalkCols / (strips + 0.5 * idle + 0.5 + (last <= 8 ? 3.5 : 0.0));
  return full >= (vec ? (R < 3 ? 0.66 : 0.82) : (R < 3 ? 0.90 : 0.945));
}

// 16-byte vectors in all planes and rows
bool walk_vec(const float* a1, const float* a2, const float* phi, const float* ref, const float* phase,
              const float* coh, int W) {
  auto vec = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  return W % 4 == 0 && vec(a1) && vec(a2) && vec(phi) && vec(ref) && vec(phase) && vec(coh);
}

template <int R>
cudaError_t launch_boxcar_walk(const float* a1, const float* a2, const float* phi, float* ref, float* phase,
                               float* coh, int H, int W, int sms, cudaStream_t st) {
  const bool all = walk_vec(a1, a2, phi, ref, phase, coh, W);
  const int gx = walk_blocks_x(W, R), rows4 = (H - 1 + R) / 4 + 1;
  // every walk sums 2 R rows before its first output: long ones where the
  // scene has several waves of them, else the length with the shortest sum of
  // waves
  const long long slots = (long long)kWalkBlocks * sms;
  int groups = kWalkGroups;
  long long best = 0;
  for (int g = kWalkGroups; g >= 1; --g) {
    const long long waves = ((long long)gx * ((rows4 + g - 1) / g) + slots - 1) / slots;
    const long long cost = waves * (4 * g + 2 * R + 4);
    if (best == 0 || cost < best) best = cost, groups = g;
  }
  const dim3 grid(gx, (rows4 + groups - 1) / groups);
  if (all)
    boxcar_walk_kernel<R, true><<<grid, 32 * kWalkWarps, 0, st>>>(a1, a2, phi, ref, phase, coh, H, W, groups);
  else
    boxcar_walk_kernel<R, false><<<grid, 32 * kWalkWarps, 0, st>>>(a1, a2, phi, ref, phase, coh, H, W, groups);
  return cudaGetLastError();
}

template <int R>
cudaError_t launch_boxcar_r(const float* a1, const float* a2, const float* phi, float* ref, float* phase, float* coh,
                            int H, int W, dim3 grid, cudaStream_t st) {
  constexpr size_t smem = (size_t)3 * ((kBoxTH + 2 * R) * ((kBoxTW + 2 * R + 3) / 4 * 4) + (kBoxTH + 2 * R) * kBoxTW) * 4;
  static size_t allowed[kMaxDevices];
  const cudaError_t e = allow_dynamic_smem((const void*)boxcar_r_kernel<R>, smem, allowed);
  if (e != cudaSuccess) return e;
  // 8-byte output vectors need an even row length and 8-byte aligned planes
  const int vec_out = (W % 2 == 0) && ((reinterpret_cast<uintptr_t>(ref) | reinterpret_cast<uintptr_t>(phase) |
                                         reinterpret_cast<uintptr_t>(coh)) % 8 == 0);
  boxcar_r_kernel<R><<<grid, kBoxThreads, smem, st>>>(a1, a2, phi, ref, phase, coh, H, W, vec_out);
  return cudaGetLastError();
}

}  // namespace

int boxcar_device(const float* a1, const float* a2, const float* phi, float* ref, float* phase, float* coh, int H,
                  int W, int w, cudaStream_t st) {
  if (!a1 || !a2 || !phi || !ref || !phase || !coh) return set_error(DCL_ERR_INVALID_ARGUMENT, "null pointer");
  if (H < 1 || W < 1) return set_error(DCL_ERR_INVALID_ARGUMENT, "height and width must be >= 1");
  if (w < 1 || w % 2 == 0 || (w - 1) / 2 > kBoxMaxR)
    return set_error(DCL_ERR_INVALID_ARGUMENT, "window width must be odd and in [1, %d], got %d", 2 * kBoxMaxR + 1, w);
  const int r = (w - 1) / 2;
  const int vH = H - 1 + r, vW = W - 1 + r;
  dim3 grid((vW + kBoxTW) / kBoxTW, (vH + kBoxTH) / kBoxTH);
  const size_t smem = (size_t)3 * ((kBoxTH + 2 * r) * (kBoxTW + 2 * r) + (kBoxTH + 2 * r) * kBoxTW) * sizeof(float);
  static size_t allowed[kMaxDevices];
  if (r > 7) {
    const cudaError_t e = allow_dynamic_smem((const void*)boxcar_kernel, smem, allowed);
    if (e != cudaSuccess) return cuda_error(e, "boxcar shared-memory limit");
  }
  // the walk has windows up to 7 x 7 (at 9 x 9 its registers leave eight warps:
  // 110 us at 4096 x 4096, tiled 114; 96 at 3000 x 4001, 92)
  const bool walk = r >= 1 && r <= 3 && walk_pays(H, W, r, walk_vec(a1, a2, phi, ref, phase, coh, W));
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = sm_count(dev);
  cudaError_t e = cudaSuccess;
  switch (r) {
    case 0: e = launch_boxcar_r<0>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 1: e = walk ? launch_boxcar_walk<1>(a1, a2, phi, ref, phase, coh, H, W, sms, st)
                       : launch_boxcar_r<1>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 2: e = walk ? launch_boxcar_walk<2>(a1, a2, phi, ref, phase, coh, H, W, sms, st)
                       : launch_boxcar_r<2>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 3: e = walk ? launch_boxcar_walk<3>(a1, a2, phi, ref, phase, coh, H, W, sms, st)
                       : launch_boxcar_r<3>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 4: e = launch_boxcar_r<4>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 5: e = launch_boxcar_r<5>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 6: e = launch_boxcar_r<6>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    case 7: e = launch_boxcar_r<7>(a1, a2, phi, ref, phase, coh, H, W, grid, st); break;
    default:
      boxcar_kernel<<<grid, kBoxThreads, smem, st>>>(a1, a2, phi, ref, phase, coh, H, W, r);
      e = cudaGetLastError();
  }
  profile_count(1);
  if (e != cudaSuccess) return cuda_error(e, "boxcar launch");
  return DCL_OK;
}

}  // namespace dcl

extern "C" int dcl_boxcar_device(const float* a1, const float* a2, const float* phi, float* ref, float* phase,
                                 float* coh, int H, int W, int window_width, void* stream) {
  return dcl::boxcar_device(a1, a2, phi, ref, phase, coh, H, W, window_width, (cudaStream_t)stream);
}

extern "C" int dcl_boxcar(const float* a1, const float* a2, const float* phi, float* ref, float* phase, float* coh,
                          int H, int W, int window_width) {
  if (!a1 || !a2 || !phi || !ref || !phase || !coh) return dcl::set_error(DCL_ERR_INVALID_ARGUMENT, "null pointer");
  if (H < 1 || W < 1) return dcl::set_error(DCL_ERR_INVALID_ARGUMENT, "height and width must be >= 1");
  cudaStream_t st = cudaStreamPerThread;
  const size_t n = (size_t)H * W, b = n * sizeof(float);
  float* buf = nullptr;
  cudaError_t e = cudaMallocAsync(&buf, 6 * b, st);
  if (e != cudaSuccess) return dcl::cuda_error(e, "cudaMallocAsync(boxcar)");
  e = cudaMemcpyAsync(buf, a1, b, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(buf + n, a2, b, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(buf + 2 * n, phi, b, cudaMemcpyHostToDevice, st);
  int rc = DCL_OK;
  if (e != cudaSuccess) rc = dcl::cuda_error(e, "cudaMemcpyAsync(H2D)");
  if (rc == DCL_OK) rc = dcl::boxcar_device(buf, buf + n, buf + 2 * n, buf + 3 * n, buf + 4 * n, buf + 5 * n, H, W,
                                            window_width, st);
  if (rc == DCL_OK) {
    e = cudaMemcpyAsync(ref, buf + 3 * n, b, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(phase, buf + 4 * n, b, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(coh, buf + 5 * n, b, cudaMemcpyDeviceToHost, st);
    if (e != cudaSuccess) rc = dcl::cuda_error(e, "cudaMemcpyAsync(D2H)");
  }
  cudaFreeAsync(buf, st);
  e = cudaStreamSynchronize(st);
  if (rc == DCL_OK && e != cudaSuccess) rc = dcl::cuda_error(e, "boxcar");
  return rc;
}

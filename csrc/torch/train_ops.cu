// Fused element-wise / normalisation / loss / optimiser kernels of the
// training step (GPT-2-style decoder, bf16 activations, fp32 arithmetic).
// The reference library has no model code at all; these kernels exist so
// that the data-parallel benchmark spends its non-GEMM time in a handful of
// bandwidth-bound passes instead of dozens of eager element-wise launches.
//
// All kernels are plain sm_100a CUDA C++: 16-byte vector accesses, one warp
// per row for the row-wise ops, grid sized as a multiple of the SM count.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>

#include "train_ops.h"
#include "train_ops_noalloc.h"
#include "device_state.h"
#include "pdl.cuh"

#include <cooperative_groups.h>
#include <mutex>

namespace cg = cooperative_groups;

namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warpMax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct alignas(16) Bf8 { bf16 v[8]; };

// Eight bf16 <-> eight floats.  The 16 bytes move as ONE 128-bit access wherever they live (global or shared memory:
// read field by field, a vector in shared memory turns into eight 2-byte loads); a bf16 is the upper half of a float.
__device__ __forceinline__ void unpack8(const Bf8 &p, float *f) {
  const uint4 u = *reinterpret_cast<const uint4 *>(&p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ Bf8 pack8(const float *f) {
  uint4 u;
  uint32_t *w = reinterpret_cast<uint32_t *>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t *>(&h);
  }
  Bf8 p;
  *reinterpret_cast<uint4 *>(&p) = u;
  return p;
}

// ---------------------------------------------------------------- LayerNorm
// One warp per row, persistent over rows, 16 warps per SM (8 for rows wider than 1024).  The rows a warp will work on
// are streamed into a private three-deep ring in shared memory with cp.async two rows ahead, so that every SM keeps
// ~128 KB of loads in flight whatever the warps are computing; a lane copies exactly the 16-byte vectors that it later reads, so
// the ring needs no barrier, only cp.async.wait_group.  C is a multiple of 256 and at most 256 * MAXV.
__device__ __forceinline__ void cpAsync16(void *smemDst, const void *gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smemDst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int MAXV, int STAGES, int LN_WARPS>
__global__ void __launch_bounds__(LN_WARPS * 32, 1) lnFwdKernel(const bf16 *x, const bf16 *delta, const bf16 *gamma, const bf16 *beta,
                                                                bf16 *resOut, bf16 *y, float *mean, float *rstd, int M, int C, float eps) {
  extern __shared__ __align__(16) uint8_t lnSmem[];
  const int warpInCta = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = blockIdx.x * LN_WARPS + warpInCta, nwarps = gridDim.x * LN_WARPS;
  const int nv = C / 256;  // 16-byte vectors per lane and row
  const int narr = delta ? 2 : 1;
  const size_t rowBytes = (size_t)C * 2;
  uint8_t *ring = lnSmem + (size_t)warpInCta * STAGES * 2 * rowBytes;
  auto issue = [&](int row, int st) {
    if (row < M) {
      uint8_t *dst = ring + (size_t)st * 2 * rowBytes;
#pragma unroll
      for (int i = 0; i < MAXV; i++)
        if (i < nv) {
          cpAsync16(dst + (i * 32 + lane) * 16, (const uint8_t *)(x + (size_t)row * C) + (i * 32 + lane) * 16);
          if (narr == 2) cpAsync16(dst + rowBytes + (i * 32 + lane) * 16, (const uint8_t *)(delta + (size_t)row * C) + (i * 32 + lane) * 16);
        }
    }
    cpAsyncCommit();  // an empty group past the last row keeps the group count uniform
  };
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
#pragma unroll
  for (int st = 0; st < STAGES - 1; st++) issue(warp + st * nwarps, st);
  int k = 0;
  for (int row = warp; row < M; row += nwarps, k++) {
    issue(row + (STAGES - 1) * nwarps, (k + STAGES - 1) % STAGES);
    cpAsyncWait<STAGES - 1>();
    const Bf8 *xr = (const Bf8 *)(ring + (size_t)(k % STAGES) * 2 * rowBytes);
    const Bf8 *dr = (const Bf8 *)((const uint8_t *)xr + rowBytes);
    float v[MAXV][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
        unpack8(xr[i * 32 + lane], v[i]);
        if (narr == 2) {
          float d[8];
          unpack8(dr[i * 32 + lane], d);
#pragma unroll
          for (int j = 0; j < 8; j++) v[i][j] += d[j];
          // the residual stream is kept in bf16: round it here so that the
          // statistics see what the next layer will read
          Bf8 r = pack8(v[i]);
          ((Bf8 *)(resOut + (size_t)row * C))[i * 32 + lane] = r;
          unpack8(r, v[i]);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) s += v[i][j];
      }
    const float mu = warpSum(s) / C;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
#pragma unroll
        for (int j = 0; j < 8; j++) { float d = v[i][j] - mu; q += d * d; }
      }
    const float rs = rsqrtf(warpSum(q) / C + eps);
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
        float g[8], b[8], o[8];
        unpack8(((const Bf8 *)gamma)[i * 32 + lane], g);
        unpack8(((const Bf8 *)beta)[i * 32 + lane], b);
#pragma unroll
        for (int j = 0; j < 8; j++) o[j] = (v[i][j] - mu) * rs * g[j] + b[j];
        ((Bf8 *)(y + (size_t)row * C))[i * 32 + lane] = pack8(o);
      }
  }
  cpAsyncWait<0>();
}

// Backward, part 1, for rows wider than 1024: dx = rstd * (g*dy - mean(g*dy) - xhat * mean(g*dy*xhat)) [+ dres].
// Same streaming scheme for dy and x; the residual gradient, needed only for the last step of a row, is loaded into
// registers when the row's turn begins.
template <int MAXV, int STAGES, int LN_WARPS>
__global__ void __launch_bounds__(LN_WARPS * 32, 1) lnBwdDxKernel(const bf16 *dy, const bf16 *x, const bf16 *gamma, const float *mean,
                                                                  const float *rstd, const bf16 *dres, bf16 *dx, int M, int C) {
  extern __shared__ __align__(16) uint8_t lnSmem[];
  const int warpInCta = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = blockIdx.x * LN_WARPS + warpInCta, nwarps = gridDim.x * LN_WARPS;
  const int nv = C / 256;
  const size_t rowBytes = (size_t)C * 2;
  uint8_t *ring = lnSmem + (size_t)warpInCta * STAGES * 2 * rowBytes;
  auto issue = [&](int row, int st) {
    if (row < M) {
      uint8_t *dst = ring + (size_t)st * 2 * rowBytes;
#pragma unroll
      for (int i = 0; i < MAXV; i++)
        if (i < nv) {
          const size_t off = (size_t)(i * 32 + lane) * 16;
          cpAsync16(dst + off, (const uint8_t *)(dy + (size_t)row * C) + off);
          cpAsync16(dst + rowBytes + off, (const uint8_t *)(x + (size_t)row * C) + off);
        }
    }
    cpAsyncCommit();
  };
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
#pragma unroll
  for (int st = 0; st < STAGES - 1; st++) issue(warp + st * nwarps, st);
  float muN = warp < M ? mean[warp] : 0.f, rsN = warp < M ? rstd[warp] : 0.f;  // statistics one row ahead
  int k = 0;
  for (int row = warp; row < M; row += nwarps, k++) {
    issue(row + (STAGES - 1) * nwarps, (k + STAGES - 1) % STAGES);
    const float mu = muN, rs = rsN;
    if (row + nwarps < M) { muN = mean[row + nwarps]; rsN = rstd[row + nwarps]; }
    Bf8 dr[MAXV];
    if (dres) {
#pragma unroll
      for (int i = 0; i < MAXV; i++)
        if (i < nv) dr[i] = ((const Bf8 *)(dres + (size_t)row * C))[i * 32 + lane];
    }
    cpAsyncWait<STAGES - 1>();
    const uint8_t *base = ring + (size_t)(k % STAGES) * 2 * rowBytes;
    const Bf8 *dyr = (const Bf8 *)base, *xr = (const Bf8 *)(base + rowBytes);
    float gy[MAXV][8], xh[MAXV][8];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
        float d[8], xv[8], g[8];
        unpack8(dyr[i * 32 + lane], d);
        unpack8(xr[i * 32 + lane], xv);
        unpack8(((const Bf8 *)gamma)[i * 32 + lane], g);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          xh[i][j] = (xv[j] - mu) * rs;
          gy[i][j] = g[j] * d[j];
          s1 += gy[i][j];
          s2 += gy[i][j] * xh[i][j];
        }
      }
    s1 = warpSum(s1) / C;
    s2 = warpSum(s2) / C;
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
        float o[8];
        if (dres) unpack8(dr[i], o);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          float t = rs * (gy[i][j] - s1 - xh[i][j] * s2);
          o[j] = dres ? o[j] + t : t;
        }
        ((Bf8 *)(dx + (size_t)row * C))[i * 32 + lane] = pack8(o);
      }
  }
  cpAsyncWait<0>();
}

// Backward in one pass over dy, x and dres for rows up to 1024 wide: dx as below, and the parameter gradients
// dgamma[c] = sum_r dy[r,c] * xhat[r,c], dbeta[c] = sum_r dy[r,c] from the values that are on chip anyway (a second kernel
// read dy and x again: 33 MB at 8192 x 1024).  The three rows of a warp stream through a ring in shared memory.  A thread
// holds 32 columns' dgamma and dbeta sums, which leaves no room for the row: it is looked at twice in shared memory, once
// for the two means and once for the results, so that sixteen warps fit on an SM (with eight that keep the row in
// registers the arithmetic set the pace: 19 us at 8192 x 1024 without the fold; with it 19.5 now, 21.6 with inputs beyond L2, where the
// two kernels that each read dy and x took 26).  At the end the warps fold their sums in shared memory and
// a CTA leaves [2][C] of them in `partial` for lnParamFoldKernel.
template <int MAXV, int STAGES, int LN_WARPS>
__global__ void __launch_bounds__(LN_WARPS * 32, 1) lnBwdFusedKernel(const bf16 *dy, const bf16 *x, const bf16 *gamma, const float *mean,
                                                                     const float *rstd, const bf16 *dres, bf16 *dx, float *partial, int M, int C) {
  extern __shared__ __align__(16) uint8_t lnSmem[];
  const int warpInCta = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = blockIdx.x * LN_WARPS + warpInCta, nwarps = gridDim.x * LN_WARPS;
  const int nv = C / 256;
  const size_t rowBytes = (size_t)C * 2;
  uint8_t *ring = lnSmem + (size_t)warpInCta * STAGES * 3 * rowBytes;
  auto issue = [&](int row, int st) {
    if (row < M) {
      uint8_t *dst = ring + (size_t)st * 3 * rowBytes;
#pragma unroll
      for (int i = 0; i < MAXV; i++)
        if (i < nv) {
          const size_t off = (size_t)(i * 32 + lane) * 16;
          cpAsync16(dst + off, (const uint8_t *)(dy + (size_t)row * C) + off);
          cpAsync16(dst + rowBytes + off, (const uint8_t *)(x + (size_t)row * C) + off);
          if (dres) cpAsync16(dst + 2 * rowBytes + off, (const uint8_t *)(dres + (size_t)row * C) + off);
        }
    }
    cpAsyncCommit();
  };
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
#pragma unroll
  for (int st = 0; st < STAGES - 1; st++) issue(warp + st * nwarps, st);
  float dg[MAXV][8], db[MAXV][8];
#pragma unroll
  for (int i = 0; i < MAXV; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) dg[i][j] = db[i][j] = 0.f;
  float muN = warp < M ? mean[warp] : 0.f, rsN = warp < M ? rstd[warp] : 0.f;  // statistics one row ahead
  int k = 0;
  for (int row = warp; row < M; row += nwarps, k++) {
    issue(row + (STAGES - 1) * nwarps, (k + STAGES - 1) % STAGES);
    const float mu = muN, rs = rsN;
    if (row + nwarps < M) { muN = mean[row + nwarps]; rsN = rstd[row + nwarps]; }
    cpAsyncWait<STAGES - 1>();
    const uint8_t *base = ring + (size_t)(k % STAGES) * 3 * rowBytes;
    const Bf8 *dyr = (const Bf8 *)base, *xr = (const Bf8 *)(base + rowBytes), *rr = (const Bf8 *)(base + 2 * rowBytes);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
        float d[8], xv[8], g[8];
        unpack8(dyr[i * 32 + lane], d);
        unpack8(xr[i * 32 + lane], xv);
        unpack8(((const Bf8 *)gamma)[i * 32 + lane], g);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float xh = (xv[j] - mu) * rs, gy = g[j] * d[j];
          s1 += gy;
          s2 += gy * xh;
          dg[i][j] += d[j] * xh;
          db[i][j] += d[j];
        }
      }
    s1 = warpSum(s1) / C;
    s2 = warpSum(s2) / C;
#pragma unroll
    for (int i = 0; i < MAXV; i++)
      if (i < nv) {
        float d[8], xv[8], g[8], o[8];
        unpack8(dyr[i * 32 + lane], d);
        unpack8(xr[i * 32 + lane], xv);
        unpack8(((const Bf8 *)gamma)[i * 32 + lane], g);
        if (dres) unpack8(rr[i * 32 + lane], o);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float t = rs * (g[j] * d[j] - s1 - (xv[j] - mu) * rs * s2);
          o[j] = dres ? o[j] + t : t;
        }
        ((Bf8 *)(dx + (size_t)row * C))[i * 32 + lane] = pack8(o);
      }
  }
  cpAsyncWait<0>();
  __syncthreads();  // the ring becomes the warps' sums: [warp][2][C]
  float *sums = (float *)lnSmem + (size_t)warpInCta * 2 * C;
#pragma unroll
  for (int i = 0; i < MAXV; i++)
    if (i < nv) {
      float4 *g4 = (float4 *)(sums + (i * 32 + lane) * 8), *b4 = (float4 *)(sums + C + (i * 32 + lane) * 8);
      g4[0] = make_float4(dg[i][0], dg[i][1], dg[i][2], dg[i][3]);
      g4[1] = make_float4(dg[i][4], dg[i][5], dg[i][6], dg[i][7]);
      b4[0] = make_float4(db[i][0], db[i][1], db[i][2], db[i][3]);
      b4[1] = make_float4(db[i][4], db[i][5], db[i][6], db[i][7]);
    }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * C; c += LN_WARPS * 32) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < LN_WARPS; w++) t += ((const float *)lnSmem)[(size_t)w * 2 * C + c];
    partial[(size_t)blockIdx.x * 2 * C + c] = t;
  }
}

// The `parts` partial sums of each of `width` columns -> one, as bf16, (+)= *target(column).  A CTA folds 32 columns with 32 warps, a
// 32nd of the parts each and up to eight loads of them in flight: the fold is a chain of memory latencies and nothing else.
// With eight warps of four loads in flight (148 parts: five turns, 296: ten) a fold kept the stream for 4.6 us in a GPT-2-medium
// step at C = 1024 (LayerNorm) and 5.4 at C = 4096 (bias of the GELU), and keeps it for 3.3 and 3.4 now.
constexpr int FOLD_WARPS = 32;
template <typename Target>
__device__ __forceinline__ void foldColumns(const float *partial, int parts, int width, int accumulate, Target target) {
  __shared__ float red[FOLD_WARPS][33];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;  // width is a multiple of 32
  float t = 0.f;
#pragma unroll 8
  for (int p = grp; p < parts; p += FOLD_WARPS) t += partial[(size_t)p * width + c];
  red[grp][lane] = t;
  __syncthreads();
  if (grp == 0) {
    t = 0.f;
#pragma unroll
    for (int g = 0; g < FOLD_WARPS; g++) t += red[g][lane];
    bf16 *dst = target(c);
    if (accumulate) t += __bfloat162float(*dst);
    *dst = __float2bfloat16_rn(t);
  }
}

// dgamma / dbeta from the [2][C] partial sums of the LayerNorm backward kernels.
__global__ void __launch_bounds__(FOLD_WARPS * 32) lnParamFoldKernel(const float *partial, int parts, int C, bf16 *dgamma, bf16 *dbeta,
                                                                     int accumulate) {
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  foldColumns(partial, parts, 2 * C, accumulate, [&](int c) { return c < C ? dgamma + c : dbeta + (c - C); });
}

// A bias gradient from the [C] partial sums of biasGeluBwdKernel.
__global__ void __launch_bounds__(FOLD_WARPS * 32) colSumFoldKernel(const float *partial, int parts, int C, bf16 *out, int accumulate) {
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  foldColumns(partial, parts, C, accumulate, [&](int c) { return out + c; });
}

// Backward, part 2, for rows wider than 1024: dgamma[c] = sum_r dy[r,c] * xhat[r,c], dbeta[c] = sum_r dy[r,c].
// A CTA owns 64 columns and one slice of the rows; partial sums go to
// `partial` ([gridDim.y][2][C], fp32 scratch), which lnParamFoldKernel folds into dgamma / dbeta.
__global__ void __launch_bounds__(256) lnBwdParamKernel(const bf16 *dy, const bf16 *x, const float *mean, const float *rstd, float *partial,
                                                        int M, int C) {
  __shared__ float redG[32][64 + 1], redB[32][64 + 1];
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  const int col0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  float dg[8] = {0, 0, 0, 0, 0, 0, 0, 0}, db[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int rowsPer = (M + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rowsPer, r1 = min(M, r0 + rowsPer);
  int r = r0 + ty;
  for (; r + 96 < r1; r += 128) {  // four rows (eight 16-byte loads) in flight per thread
    Bf8 pd[4], px[4];
    float m[4], sd[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      pd[u] = *(const Bf8 *)(dy + (size_t)(r + 32 * u) * C + col0 + tx * 8);
      px[u] = *(const Bf8 *)(x + (size_t)(r + 32 * u) * C + col0 + tx * 8);
      m[u] = mean[r + 32 * u];
      sd[u] = rstd[r + 32 * u];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      float d0[8], x0[8];
      unpack8(pd[u], d0);
      unpack8(px[u], x0);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        dg[k] += d0[k] * (x0[k] - m[u]) * sd[u];
        db[k] += d0[k];
      }
    }
  }
  for (; r < r1; r += 32) {
    float d0[8], x0[8];
    unpack8(*(const Bf8 *)(dy + (size_t)r * C + col0 + tx * 8), d0);
    unpack8(*(const Bf8 *)(x + (size_t)r * C + col0 + tx * 8), x0);
    const float m0 = mean[r], s0 = rstd[r];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      dg[k] += d0[k] * (x0[k] - m0) * s0;
      db[k] += d0[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 8; k++) { redG[ty][tx * 8 + k] = dg[k]; redB[ty][tx * 8 + k] = db[k]; }
  __syncthreads();
  if (threadIdx.x < 128) {
    const int c = threadIdx.x & 63;
    const bool isB = threadIdx.x >= 64;
    float s = 0.f;
#pragma unroll 8
    for (int j = 0; j < 32; j++) s += isB ? redB[j][c] : redG[j][c];
    partial[((size_t)blockIdx.y * 2 + (isB ? 1 : 0)) * C + col0 + c] = s;
  }
}

// ---------------------------------------------------------------- bias + GELU (tanh form)
__device__ __forceinline__ float fastTanh(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float geluF(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.f + fastTanh(k0 * (x + k1 * x * x * x)));
}
__device__ __forceinline__ float geluGrad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x), t = fastTanh(u);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
}

// y = gelu(x + bias); x is [M, C].  Each thread keeps four 16-byte loads in flight.
__global__ void __launch_bounds__(256) biasGeluFwdKernel(const bf16 *x, const bf16 *bias, bf16 *y, size_t nvec, int C) {
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  const int cv = C / 8;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < nvec; i += 4 * stride) {
    Bf8 v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = ((const Bf8 *)x)[i + j * stride];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float a[8], b[8];
      unpack8(v[j], a);
      unpack8(((const Bf8 *)bias)[(i + j * stride) % cv], b);
#pragma unroll
      for (int k = 0; k < 8; k++) a[k] = geluF(a[k] + b[k]);
      ((Bf8 *)y)[i + j * stride] = pack8(a);
    }
  }
  for (; i < nvec; i += stride) {
    float a[8], b[8];
    unpack8(((const Bf8 *)x)[i], a);
    unpack8(((const Bf8 *)bias)[i % cv], b);
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = geluF(a[k] + b[k]);
    ((Bf8 *)y)[i] = pack8(a);
  }
}

// dx = dy * gelu'(x + bias) and, from the same values, the partial column sums of the bias gradient ([gridDim.y][C], fp32,
// folded by colSumFoldKernel).  A CTA owns VX * 8 columns (all 256 threads side by side on wide rows) and every gridDim.y-th
// group of 256 / VX rows, four rows (eight 16-byte loads) in flight per thread; a thread keeps its eight columns throughout.
// Bound by memory (dy, x, dx: 201 MB and 30 us at 8192 x 4096) with the arithmetic close behind.  Blocks of 64 columns with a
// fold in the last CTA took 55 us: their CTAs lived for eight rows per thread.  With the fold kernel 49 us (53 while its pointers were
// restrict-qualified).
__global__ void __launch_bounds__(256) biasGeluBwdKernel(const bf16 *dy, const bf16 *x, const bf16 *bias, bf16 *dx, float *partial, int M, int C,
                                                         int VX) {
  __shared__ float red[2048];
  const int tx = threadIdx.x % VX, ty = threadIdx.x / VX, RY = 256 / VX;
  const int col = (blockIdx.x * VX + tx) * 8;
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, b[8];
  unpack8(*(const Bf8 *)(bias + col), b);
  auto one = [&](const Bf8 &xv, const Bf8 &dv, size_t off) {
    float a[8], d[8];
    unpack8(xv, a);
    unpack8(dv, d);
#pragma unroll
    for (int k = 0; k < 8; k++) d[k] *= geluGrad(a[k] + b[k]);
    const Bf8 o = pack8(d);
    *(Bf8 *)(dx + off) = o;
    unpack8(o, d);  // the sum is that of the stored gradient
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] += d[k];
  };
  const int step = gridDim.y * RY;
  int r = blockIdx.y * RY + ty;
  for (; r + 3 * step < M; r += 4 * step) {
    Bf8 xv[4], dv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const size_t off = (size_t)(r + u * step) * C + col;
      xv[u] = *(const Bf8 *)(x + off);
      dv[u] = *(const Bf8 *)(dy + off);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) one(xv[u], dv[u], (size_t)(r + u * step) * C + col);
  }
  for (; r < M; r += step) {
    const size_t off = (size_t)r * C + col;
    one(*(const Bf8 *)(x + off), *(const Bf8 *)(dy + off), off);
  }
  // fold the row lanes of the CTA, then one sum per column
#pragma unroll
  for (int k = 0; k < 8; k++) red[(ty * VX + tx) * 8 + k] = acc[k];
  __syncthreads();
  for (int c = threadIdx.x; c < VX * 8; c += 256) {
    float t = 0.f;
    for (int y = 0; y < RY; y++) t += red[y * VX * 8 + c];
    partial[(size_t)blockIdx.y * C + blockIdx.x * VX * 8 + c] = t;
  }
}

// Column sums of a [M, C] bf16 matrix (bias gradients).  Each CTA owns 64
// columns and a slice of rows; partials go to fp32 scratch [gridDim.y][C].
__global__ void __launch_bounds__(256) colSumKernel(const bf16 *__restrict__ a, float *__restrict__ partial, int M, int C) {
  const int col0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;  // 8 vector columns x 32 row lanes
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int rowsPer = (M + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rowsPer, r1 = min(M, r0 + rowsPer);
  int r = r0 + ty;
  for (; r + 96 < r1; r += 128) {  // four rows in flight per thread
    Bf8 p[4];
#pragma unroll
    for (int u = 0; u < 4; u++) p[u] = *(const Bf8 *)(a + (size_t)(r + 32 * u) * C + col0 + tx * 8);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      float v[8];
      unpack8(p[u], v);
#pragma unroll
      for (int k = 0; k < 8; k++) acc[k] += v[k];
    }
  }
  for (; r < r1; r += 32) {
    float v[8];
    unpack8(*(const Bf8 *)(a + (size_t)r * C + col0 + tx * 8), v);
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] += v[k];
  }
  // reduce over the 32 row lanes: lanes with equal tx live in different warps, go through shared memory
  __shared__ float red[32][64 + 1];
#pragma unroll
  for (int k = 0; k < 8; k++) red[ty][tx * 8 + k] = acc[k];
  __syncthreads();
  if (threadIdx.x < 64) {
    float s = 0.f;
#pragma unroll 8
    for (int j = 0; j < 32; j++) s += red[j][threadIdx.x];
    partial[(size_t)blockIdx.y * C + col0 + threadIdx.x] = s;
  }
}

__global__ void colSumReduceKernel(const float *__restrict__ partial, int nparts, int C, bf16 *__restrict__ out, int accumulate) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float s = 0.f;
  for (int p = 0; p < nparts; p++) s += partial[(size_t)p * C + c];
  if (accumulate) s += __bfloat162float(out[c]);
  out[c] = __float2bfloat16_rn(s);
}

// The column sums in ONE launch.  A CTA owns 64 columns and a slice of the rows; the CTAs of a column block form a cluster
// (up to eight), whose first CTA adds up the others' sums out of their shared memory.  Nothing outlives the launch, so calls
// on several streams do not meet; with tickets in the library image, as this kernel had before, concurrent calls of a device
// took each other's.  Bound by memory once there are rows enough, by latency below.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) colSumClusterKernel(const bf16 *a, bf16 *out, int M, int C, int accumulate) {
  constexpr int ROWS = THREADS / 8, WARPS = THREADS / 32;
  __shared__ float red[WARPS][64], sums[64];
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  const int col0 = blockIdx.x * 64, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;  // 8 vector columns x ROWS row lanes
  const int rowsPer = (M + gridDim.y - 1) / gridDim.y;
  const int r1 = min(M, (int)(blockIdx.y + 1) * rowsPer);
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int r = blockIdx.y * rowsPer + ty; r < r1; r += 4 * ROWS) {  // four rows in flight per thread
    Bf8 p[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (r + u * ROWS < r1) p[u] = *(const Bf8 *)(a + (size_t)(r + u * ROWS) * C + col0 + tx * 8);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (r + u * ROWS < r1) {
        float v[8];
        unpack8(p[u], v);
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] += v[k];
      }
  }
#pragma unroll
  for (int k = 0; k < 8; k++) {  // the four rows of a warp
    acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 8);
    acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 16);
  }
  if (lane < 8) {
#pragma unroll
    for (int k = 0; k < 8; k++) red[warp][lane * 8 + k] = acc[k];
  }
  __syncthreads();
  float s = 0.f;
  if (threadIdx.x < 64) {
#pragma unroll
    for (int w = 0; w < WARPS; w++) s += red[w][threadIdx.x];
    sums[threadIdx.x] = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (blockIdx.y == 0 && threadIdx.x < 64) {
    for (unsigned int i = 1; i < gridDim.y; i++) s += *cluster.map_shared_rank(&sums[threadIdx.x], i);
    bf16 *dst = out + col0 + threadIdx.x;
    if (accumulate) s += __bfloat162float(*dst);
    *dst = __float2bfloat16_rn(s);
  }
  cluster.sync();  // nobody's shared memory goes before it has been read
}

// ---------------------------------------------------------------- softmax cross-entropy
// One CTA per row of logits [M, Vpad] (V valid columns).  Writes the loss of
// the row and overwrites the logits with (softmax - onehot) * gradScale.
__global__ void __launch_bounds__(1024) ceFwdBwdKernel(bf16 *__restrict__ logits, const int64_t *__restrict__ targets,
                                                       float *__restrict__ losses, int V, int Vpad, float gradScale) {
  __shared__ float red[32];
  __shared__ float bcast;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  bf16 *lr = logits + (size_t)row * Vpad;
  const int nvec = V / 8;
  const int tgt = (int)targets[row];
  // read before anything in the row is overwritten by the gradient pass
  const float tgtLogit = (tgt >= 0 && tgt < V) ? __bfloat162float(lr[tgt]) : 0.f;
  float mx = -INFINITY;
  for (int i = tid; i < nvec; i += blockDim.x) {
    float v[8];
    unpack8(((const Bf8 *)lr)[i], v);
#pragma unroll
    for (int k = 0; k < 8; k++) mx = fmaxf(mx, v[k]);
  }
  for (int i = nvec * 8 + tid; i < V; i += blockDim.x) mx = fmaxf(mx, __bfloat162float(lr[i]));
  mx = warpMax(mx);
  if (lane == 0) red[wid] = mx;
  __syncthreads();
  if (wid == 0) {
    float v = lane < nw ? red[lane] : -INFINITY;
    v = warpMax(v);
    if (lane == 0) bcast = v;
  }
  __syncthreads();
  mx = bcast;
  float sum = 0.f;
  for (int i = tid; i < nvec; i += blockDim.x) {
    float v[8];
    unpack8(((const Bf8 *)lr)[i], v);
#pragma unroll
    for (int k = 0; k < 8; k++) sum += __expf(v[k] - mx);
  }
  for (int i = nvec * 8 + tid; i < V; i += blockDim.x) sum += __expf(__bfloat162float(lr[i]) - mx);
  sum = warpSum(sum);
  __syncthreads();
  if (lane == 0) red[wid] = sum;
  __syncthreads();
  if (wid == 0) {
    float v = lane < nw ? red[lane] : 0.f;
    v = warpSum(v);
    if (lane == 0) bcast = v;
  }
  __syncthreads();
  sum = bcast;
  const float inv = 1.f / sum;
  if (tid == 0) losses[row] = tgt >= 0 ? (logf(sum) + mx - tgtLogit) : 0.f;
  const float gs = tgt >= 0 ? gradScale : 0.f;
  for (int i = tid; i < nvec; i += blockDim.x) {
    float v[8];
    unpack8(((const Bf8 *)lr)[i], v);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      float p = __expf(v[k] - mx) * inv;
      v[k] = (p - ((i * 8 + k) == tgt ? 1.f : 0.f)) * gs;
    }
    ((Bf8 *)lr)[i] = pack8(v);
  }
  for (int i = nvec * 8 + tid; i < Vpad; i += blockDim.x) {
    float g = 0.f;
    if (i < V) g = (__expf(__bfloat162float(lr[i]) - mx) * inv - (i == tgt ? 1.f : 0.f)) * gs;
    lr[i] = __float2bfloat16_rn(g);
  }
}

// The same for rows that fit twice into shared memory (Vpad <= 56 K): persistent CTAs, one per SM, walk the rows; the
// row a CTA works on lies in shared memory, and the next row streams in with cp.async during the three passes over the
// current one, so the logits are read from DRAM exactly once and the reads never wait for the arithmetic.  A thread
// copies exactly the vectors it reads itself, so the only synchronisation of the ring is cp.async.wait_group.
__global__ void __launch_bounds__(1024, 1) ceFwdBwdStreamKernel(bf16 *logits, const int64_t *targets, float *losses, int M, int V, int Vpad,
                                                                float gradScale) {
  extern __shared__ __align__(16) uint8_t ceSmem[];
  __shared__ float red[2][32];
  __shared__ float bcast[2];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nvecPad = Vpad / 8;
  const size_t rowBytes = (size_t)Vpad * 2;
  auto issue = [&](int row, int b) {
    if (row < M) {
      const uint8_t *src = (const uint8_t *)(logits + (size_t)row * Vpad);
      uint8_t *dst = ceSmem + (size_t)b * rowBytes;
      for (int i = tid; i < nvecPad; i += 1024) cpAsync16(dst + (size_t)i * 16, src + (size_t)i * 16);
    }
    cpAsyncCommit();
  };
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  issue(blockIdx.x, 0);
  int k = 0;
  for (int row = blockIdx.x; row < M; row += gridDim.x, k++) {
    issue(row + gridDim.x, (k + 1) & 1);
    bf16 *lr = logits + (size_t)row * Vpad;
    const int tgt = (int)targets[row];
    const float tgtLogit = (tgt >= 0 && tgt < V) ? __bfloat162float(lr[tgt]) : 0.f;  // before the row is overwritten
    cpAsyncWait<1>();
    Bf8 *sr = (Bf8 *)(ceSmem + (size_t)(k & 1) * rowBytes);
    // pass 1: row maximum, on packed bf16 pairs
    __nv_bfloat162 mx2 = __floats2bfloat162_rn(-INFINITY, -INFINITY);
    float mx = -INFINITY;
    for (int i = tid; i < V / 8; i += 1024) {
      const Bf8 pv = sr[i];
      const __nv_bfloat162 *h = (const __nv_bfloat162 *)&pv;
#pragma unroll
      for (int j = 0; j < 4; j++) mx2 = __hmax2(mx2, h[j]);
    }
    for (int i = V / 8 + tid; i < nvecPad; i += 1024) {
      float v[8];
      unpack8(sr[i], v);
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (i * 8 + j < V) mx = fmaxf(mx, v[j]);
    }
    mx = fmaxf(mx, fmaxf(__low2float(mx2), __high2float(mx2)));
    mx = warpMax(mx);
    if (lane == 0) red[0][wid] = mx;
    __syncthreads();
    if (wid == 0) {
      float v = warpMax(red[0][lane]);
      if (lane == 0) bcast[0] = v;
    }
    __syncthreads();
    mx = bcast[0];
    // pass 2: e = exp(v - max), summed in fp32 and left in the row buffer as bf16 (columns past V become 0), so that
    // the gradient pass needs no second exponential
    const float kLog2e = 1.4426950408889634f, mxl = mx * kLog2e;
    float sum = 0.f, sumB = 0.f;
    const int nvecFull = V / 8;
    for (int i = tid; i < nvecFull; i += 1024) {  // whole vectors: no masks, two independent partial sums
      float v[8];
      unpack8(sr[i], v);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fmaf(v[j], kLog2e, -mxl)));
        if (j & 1) sumB += e; else sum += e;
        v[j] = e;
      }
      sr[i] = pack8(v);
    }
    for (int i = nvecFull + tid; i < nvecPad; i += 1024) {  // the ragged vector and the padding behind it
      float v[8];
      unpack8(sr[i], v);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float e = 0.f;
        if (i * 8 + j < V) asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(fmaf(v[j], kLog2e, -mxl)));
        sum += e;
        v[j] = e;
      }
      sr[i] = pack8(v);
    }
    sum += sumB;
    sum = warpSum(sum);
    if (lane == 0) red[1][wid] = sum;
    __syncthreads();
    if (wid == 0) {
      float v = warpSum(red[1][lane]);
      if (lane == 0) bcast[1] = v;
    }
    __syncthreads();
    sum = bcast[1];
    if (tid == 0) losses[row] = tgt >= 0 ? (logf(sum) + mx - tgtLogit) : 0.f;
    // pass 3: gradient = (e / sum - onehot) * scale
    const float gs = tgt >= 0 ? gradScale : 0.f, scale = gs / sum;
    const int tgtVec = (tgt >= 0 && tgt < V) ? (tgt >> 3) : -1;
    for (int i = tid; i < nvecPad; i += 1024) {
      float v[8];
      unpack8(sr[i], v);
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] *= scale;
      ((Bf8 *)lr)[i] = pack8(v);
    }
    // the target column, by the thread that stored the vector around it a moment ago
    if (tgtVec >= 0 && (tgtVec & 1023) == tid)
      lr[tgt] = __float2bfloat16_rn(__bfloat162float(((const bf16 *)sr)[tgt]) * scale - gs);
    // red / bcast are rewritten only after the next row's first barrier pair; nothing else is shared between rows
  }
  cpAsyncWait<0>();
}

// ---------------------------------------------------------------- AdamW on flat buffers
// master (fp32) is the truth; param (bf16) is refreshed from it.  The gradient
// is read once and cleared, so no separate zero_grad pass is needed.
__global__ void __launch_bounds__(256) adamwKernel(float *master, bf16 *param, bf16 *grad, float *m, float *v, size_t n, float lr, float b1,
                                                   float b2, float eps, float wd, float bc1, float bc2, float gradScale, int zeroGrad,
                                                   const int *stepDev) {
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  if (stepDev) {
    // step counter kept on the device so that a captured graph stays exact
    float st = (float)(*stepDev);
    bc1 = 1.f - powf(b1, st);
    bc2 = 1.f - powf(b2, st);
  }
  const size_t nvec = n / 8;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) {
    float g[8];
    unpack8(((const Bf8 *)grad)[i], g);
    float4 w0 = ((float4 *)master)[2 * i], w1 = ((float4 *)master)[2 * i + 1];
    float4 m0 = ((float4 *)m)[2 * i], m1 = ((float4 *)m)[2 * i + 1];
    float4 v0 = ((float4 *)v)[2 * i], v1 = ((float4 *)v)[2 * i + 1];
    float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
    float mm[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
    float vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
    for (int k = 0; k < 8; k++) {
      float gk = g[k] * gradScale;
      mm[k] = b1 * mm[k] + (1.f - b1) * gk;
      vv[k] = b2 * vv[k] + (1.f - b2) * gk * gk;
      float upd = (mm[k] / bc1) / (sqrtf(vv[k] / bc2) + eps);
      w[k] = w[k] - lr * (upd + wd * w[k]);
    }
    ((float4 *)master)[2 * i] = make_float4(w[0], w[1], w[2], w[3]);
    ((float4 *)master)[2 * i + 1] = make_float4(w[4], w[5], w[6], w[7]);
    ((float4 *)m)[2 * i] = make_float4(mm[0], mm[1], mm[2], mm[3]);
    ((float4 *)m)[2 * i + 1] = make_float4(mm[4], mm[5], mm[6], mm[7]);
    ((float4 *)v)[2 * i] = make_float4(vv[0], vv[1], vv[2], vv[3]);
    ((float4 *)v)[2 * i + 1] = make_float4(vv[4], vv[5], vv[6], vv[7]);
    ((Bf8 *)param)[i] = pack8(w);
    if (zeroGrad) {
      Bf8 z;
#pragma unroll
      for (int k = 0; k < 8; k++) z.v[k] = __float2bfloat16_rn(0.f);
      ((Bf8 *)grad)[i] = z;
    }
  }
  // tail (n not a multiple of 8)
  if (blockIdx.x == 0) {
    for (size_t i = nvec * 8 + threadIdx.x; i < n; i += blockDim.x) {
      float gk = __bfloat162float(grad[i]) * gradScale;
      float mk = b1 * m[i] + (1.f - b1) * gk, vk = b2 * v[i] + (1.f - b2) * gk * gk;
      float wk = master[i];
      wk = wk - lr * ((mk / bc1) / (sqrtf(vk / bc2) + eps) + wd * wk);
      m[i] = mk; v[i] = vk; master[i] = wk;
      param[i] = __float2bfloat16_rn(wk);
      if (zeroGrad) grad[i] = __float2bfloat16_rn(0.f);
    }
  }
}

using fcxhost::smCount;

}  // namespace

// ---------------------------------------------------------------- launchers

extern "C" {

static int lnParts(int M) { return max(1, min(32, M / 128)); }
constexpr int LN_BWD_WARPS = 16;
static int lnFusedGrid(int M) { return std::max(1, std::min(smCount(), (M + LN_BWD_WARPS - 1) / LN_BWD_WARPS)); }
int fcxLnPartials(int M) { return std::max(lnParts(M), lnFusedGrid(M)); }

cudaError_t fcxLayerNormFwd(const void *x, const void *delta, const void *gamma, const void *beta, void *resOut, void *y,
                            float *mean, float *rstd, int M, int C, float eps, cudaStream_t s) {
  if (C % 256 != 0 || C > 256 * 8) return cudaErrorInvalidValue;
  // rows up to 1024 wide: 16 warps per SM (the arithmetic needs the issue slots), wider rows: 8 warps; either way
  // warps x 3-deep ring x (x, delta) x row bytes <= 192 KB
  const int warps = C <= 1024 ? 16 : 8;
  const int grid = std::max(1, std::min(smCount(), (M + warps - 1) / warps));
  const size_t smem = (size_t)warps * 3 * 2 * C * 2;
  auto run = [&](auto kernel) {
    // both instantiations have the same pointer type, so this lambda exists once: one entry for each
    static fcxhost::OncePerDevice once[2];
    const cudaError_t e = once[warps == 8]([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
    if (e != cudaSuccess) return e;
    return fcxpdl::launchPdl(kernel, grid, warps * 32, smem, s, (const bf16 *)x, (const bf16 *)delta, (const bf16 *)gamma, (const bf16 *)beta,
                             (bf16 *)resOut, (bf16 *)y, mean, rstd, M, C, eps);
  };
  return C <= 1024 ? run(lnFwdKernel<4, 3, 16>) : run(lnFwdKernel<8, 3, 8>);
}

// `partial` must hold fcxLnPartials(M) * 2 * C floats.
cudaError_t fcxLayerNormBwd(const void *dy, const void *x, const void *gamma, const float *mean, const float *rstd,
                            const void *dres, void *dx, void *dgamma, void *dbeta, float *partial, int M, int C, int accumulate,
                            cudaStream_t s) {
  if (C % 256 != 0 || C > 256 * 8) return cudaErrorInvalidValue;
  if (C <= 1024) {
    constexpr int STAGES = 2, WARPS = LN_BWD_WARPS;
    const size_t smem = (size_t)WARPS * STAGES * 3 * C * 2;  // at most 192 KB; the warps' sums (WARPS x 2 x C fp32) fit in it
    auto kernel = lnBwdFusedKernel<4, STAGES, WARPS>;
    static fcxhost::OncePerDevice once;
    cudaError_t e = once([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
    if (e != cudaSuccess) return e;
    const int grid = lnFusedGrid(M);
    e = fcxpdl::launchPdl(kernel, grid, WARPS * 32, smem, s, (const bf16 *)dy, (const bf16 *)x, (const bf16 *)gamma, mean, rstd,
                                      (const bf16 *)dres, (bf16 *)dx, partial, M, C);
    if (e != cudaSuccess) return e;
    return fcxpdl::launchPdl(lnParamFoldKernel, 2 * C / 32, FOLD_WARPS * 32, 0, s, (const float *)partial, grid, C, (bf16 *)dgamma, (bf16 *)dbeta, accumulate);
  }
  constexpr int WARPS = 8;
  const size_t smem = (size_t)WARPS * 3 * 2 * C * 2;  // warps x 3-deep ring x (dy, x) x row bytes <= 192 KB
  auto kernel = lnBwdDxKernel<8, 3, WARPS>;
  static fcxhost::OncePerDevice once;
  cudaError_t e = once([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
  if (e != cudaSuccess) return e;
  e = fcxpdl::launchPdl(kernel, std::max(1, std::min(smCount(), (M + WARPS - 1) / WARPS)), WARPS * 32, smem, s, (const bf16 *)dy,
                                    (const bf16 *)x, (const bf16 *)gamma, mean, rstd, (const bf16 *)dres, (bf16 *)dx, M, C);
  if (e != cudaSuccess) return e;
  const int parts = lnParts(M);
  e = fcxpdl::launchPdl(lnBwdParamKernel, dim3(C / 64, parts), 256, 0, s, (const bf16 *)dy, (const bf16 *)x, mean, rstd, partial, M, C);
  if (e != cudaSuccess) return e;
  return fcxpdl::launchPdl(lnParamFoldKernel, 2 * C / 32, FOLD_WARPS * 32, 0, s, (const float *)partial, parts, C, (bf16 *)dgamma, (bf16 *)dbeta, accumulate);
}

cudaError_t fcxBiasGeluFwd(const void *x, const void *bias, void *y, size_t M, int C, cudaStream_t s) {
  if (C % 8 != 0) return cudaErrorInvalidValue;
  size_t nvec = M * C / 8;
  int grid = (int)std::min<size_t>((nvec + 255) / 256, (size_t)smCount() * 8);
  return fcxpdl::launchPdl(biasGeluFwdKernel, grid, 256, 0, s, (const bf16 *)x, (const bf16 *)bias, (bf16 *)y, nvec, C);
}

int fcxColSumPartials(int M) { return max(1, min(32, M / 256)); }

// Eight-column vectors that a CTA of biasGeluBwdKernel covers side by side, and its number of row groups.
static void biasGeluBwdShape(int M, int C, int *vx, int *parts) {
  const int cv = C / 8;
  *vx = 256;
  while (cv % *vx) *vx /= 2;  // C is a multiple of 64: 8 at least
  const int rows = 256 / *vx, blocks = cv / *vx;
  *parts = std::max(1, std::min((M + 4 * rows - 1) / (4 * rows), (4 * smCount() + blocks - 1) / blocks));
}

int fcxBiasGeluBwdPartials(int M, int C) {
  int vx = 0, parts = 0;
  if (C % 64 != 0 || C <= 0) return 1;
  biasGeluBwdShape(M, C, &vx, &parts);
  return parts;
}

cudaError_t fcxBiasGeluBwd(const void *dy, const void *x, const void *bias, void *dx, void *dbias, float *partial, int M, int C,
                           int accumulate, cudaStream_t s) {
  if (C % 64 != 0) return cudaErrorInvalidValue;
  int vx = 0, parts = 0;
  biasGeluBwdShape(M, C, &vx, &parts);
  cudaError_t e = fcxpdl::launchPdl(biasGeluBwdKernel, dim3(C / 8 / vx, parts), 256, 0, s, (const bf16 *)dy, (const bf16 *)x, (const bf16 *)bias,
                                    (bf16 *)dx, partial, M, C, vx);
  if (e != cudaSuccess) return e;
  return fcxpdl::launchPdl(colSumFoldKernel, C / 32, FOLD_WARPS * 32, 0, s, (const float *)partial, parts, C, (bf16 *)dbias, accumulate);
}

cudaError_t fcxColSum(const void *a, void *out, int M, int C, int accumulate, cudaStream_t s) {
  if (C % 64 != 0) return cudaErrorInvalidValue;
  // A CTA for every 256 rows, up to the eight of a portable cluster.  From 1024 rows on, CTAs of 512 threads while they all fit
  // on the SMs at once (three each): in microseconds, 256 / 512 threads, 2328 x 2944 6.6 / 6.0, 8192 x 1024 9.9 / 7.8,
  // 8192 x 3072 12.8 / 11.0, but 8192 x 4096 (512 CTAs) 13.8 / 18.0 and 64 x 3072 2.3 / 2.5.  (With tickets: 7.5, 7.6, 14.2, 15.8, 3.1.)
  int parts = 1;
  while (parts < 8 && parts * 512 <= M) parts *= 2;
  auto run = [&](auto kernel, int threads) {
    return fcxpdl::launchPdlCluster(kernel, dim3(C / 64, parts), threads, dim3(1, parts), s, (const bf16 *)a, (bf16 *)out, M, C, accumulate);
  };
  return M >= 1024 && C / 64 * parts <= 3 * smCount() ? run(colSumClusterKernel<512>, 512) : run(colSumClusterKernel<256>, 256);
}

cudaError_t fcxCrossEntropyFwdBwd(void *logits, const int64_t *targets, float *losses, int M, int V, int Vpad, float gradScale,
                                  cudaStream_t s) {
  if (Vpad % 8 != 0 || V > Vpad) return cudaErrorInvalidValue;
  const size_t ring = (size_t)Vpad * 2 * 2;
  if (ring <= 224 * 1024 && ((uintptr_t)logits & 15) == 0) {
    static fcxhost::OncePerDevice once;
    const cudaError_t e = once([] { return cudaFuncSetAttribute(ceFwdBwdStreamKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024); });
    if (e != cudaSuccess) return e;
    return fcxpdl::launchPdl(ceFwdBwdStreamKernel, std::min(M, smCount()), 1024, ring, s, (bf16 *)logits, targets, losses, M, V, Vpad, gradScale);
  } else {
    ceFwdBwdKernel<<<M, 1024, 0, s>>>((bf16 *)logits, targets, losses, V, Vpad, gradScale);
  }
  return cudaGetLastError();
}

cudaError_t fcxAdamW(float *master, void *param, void *grad, float *m, float *v, size_t n, float lr, float b1, float b2, float eps,
                     float wd, int step, float gradScale, int zeroGrad, const int *stepDev, cudaStream_t s) {
  float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  int grid = (int)std::min<size_t>((n / 8 + 255) / 256 + 1, (size_t)smCount() * 8);
  return fcxpdl::launchPdl(adamwKernel, grid, 256, 0, s, master, (bf16 *)param, (bf16 *)grad, m, v, n, lr, b1, b2, eps, wd, bc1, bc2, gradScale,
                           zeroGrad, stepDev);
}

}  // extern "C"

// ---------------------------------------------------------------- allocation-free column sum
// (contract in train_ops_noalloc.h)

// Scratch that belongs to the library image.  In host code this name is only
// a handle for the runtime; the address a kernel can use is obtained with
// cudaGetSymbolAddress below.
static __device__ __align__(256) float gNoAllocScratch[FCX_NOALLOC_MAX_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
float *gScratchAddr[kMaxDevices];
std::mutex gScratchMu;

// Device address of the scratch array on the current device, looked up once per device.
int scratchForCurrentDevice(float **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return (int)cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(gScratchMu);
  if (!gScratchAddr[dev]) {
    float *p = nullptr;
    e = cudaGetSymbolAddress((void **)&p, gNoAllocScratch);
    if (e != cudaSuccess) return (int)e;
    gScratchAddr[dev] = p;
  }
  *out = gScratchAddr[dev];
  return 0;
}
}  // namespace

extern "C" int fcxColSumNoAlloc(const void *a, void *out, int M, int C, int accumulate, cudaStream_t stream) {
  if (!a || !out) return FCX_NOALLOC_NULL_POINTER;
  if (M <= 0 || C <= 0 || C % 64 != 0) return FCX_NOALLOC_BAD_SHAPE;
  // the kernels read `a` in 16-byte vectors; a raw-pointer caller with an odd offset gets a code, not a fault
  if (((uintptr_t)a & 15u) != 0 || ((uintptr_t)out & 15u) != 0) return FCX_NOALLOC_MISALIGNED;
  const int parts = fcxColSumPartials(M);
  if ((long long)parts * C > (long long)FCX_NOALLOC_MAX_FLOATS) return FCX_NOALLOC_TOO_LARGE;
  float *scratch = nullptr;
  int rc = scratchForCurrentDevice(&scratch);
  if (rc != 0) return rc;
  // Every partial[p][c] with p < parts, c < C is written by colSumKernel before
  // colSumReduceKernel reads it, so stale contents of earlier calls are harmless.
  colSumKernel<<<dim3(C / 64, parts), 256, 0, stream>>>((const bf16 *)a, scratch, M, C);
  colSumReduceKernel<<<(C + 255) / 256, 256, 0, stream>>>(scratch, parts, C, (bf16 *)out, accumulate);
  return (int)cudaGetLastError();
}

extern "C" const char *fcxNoAllocErrorString(int code) {
  switch (code) {
    case 0: return "success";
    case FCX_NOALLOC_TOO_LARGE: return "shape needs more than the built-in scratch (partials x C > 262144 floats); use fcxColSum";
    case FCX_NOALLOC_BAD_SHAPE: return "M and C must be positive and C a multiple of 64";
    case FCX_NOALLOC_NULL_POINTER: return "input and output pointers must not be null";
    case FCX_NOALLOC_MISALIGNED: return "input and output pointers must be 16-byte aligned";
    default: return code > 0 ? cudaGetErrorString((cudaError_t)code) : "unknown code";
  }
}

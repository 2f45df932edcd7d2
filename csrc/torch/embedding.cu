// Token + position embedding of the decoder, forward and backward.
//
//   forward   x[i] = wte[tokens[i]] + wpe[i % T]                               one warp per row
//   backward  dwte[t] += sum of dx[i] over the positions i that hold token t    (fp32 sums in position order, one rounding)
//             dwpe[p] += sum of dx[i] over the batch
//
// The backward pass adds straight into the gradients, touching only the rows whose tokens occur.  Through the library's
// embedding a GPT-2-medium step sorted the tokens (eight radix passes over 64-bit keys), wrote a dense zeroed 103 MB gradient,
// scattered into it and added it to the one that the output projection had left: forward and backward 350 us of a step of 8 x
// 1024 tokens and 215 of one of 3 x 776, 67 and 20 now, and eight launches fewer in a step of the smallest model.
//
// Duplicates are found by looking at all M tokens, which lie in shared memory as 32-bit numbers, 128 at a time: a position
// whose token occurred before is skipped, the first one collects all of its rows.  That is M^2 / 128 steps of a warp, little
// beside the rows themselves up to the EMB_MAX_TOKENS positions that the caller keeps to.  A token with many rows (punctuation) is
// left to the whole CTA, whose warps take a stretch of the positions each, and one that holds a good part of all positions
// (padding) to a pair of CTAs, whose warps take every 32nd position each: one SM alone reads about 100 GB/s.
// Forward and backward, library / one CTA for every token / so, us: 16 x 1024 positions of one token, 2048 columns 570 / 790 / 389; 8
// x 1024 x 1024, half of the positions one token, 328 / 177 / 78 (256 tokens in the table 165 / 188 / 69).
//
// The reference has no model code; this serves the data-parallel benchmark's decoder.
#include <algorithm>
#include <cassert>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_state.h"
#include "embedding.h"
#include "pdl.cuh"

namespace cg = cooperative_groups;

namespace {

using bf16 = __nv_bfloat16;

constexpr int WARPS = 16;
constexpr int HEAVY = 8;         // more rows than this are the whole CTA's work
constexpr int HEAVY_LIST = 128;  // heavy tokens of one CTA; one that finds the list full is worked on by its warp alone
// More rows than this, and than a quarter of all, are the work of a pair of CTAs.  Fewer, or more of such tokens, are as soon done by
// one CTA each (8 tokens of 1024 rows of 1024: 49 us, 69 by pairs; 1164 rows 50 and 56).
constexpr int PAIRED = 2048;

__device__ __forceinline__ void addRow(float *acc, const uint4 &u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    acc[2 * i] += __uint_as_float(w[i] << 16);  // a bf16 is the upper half of a float
    acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 packRow(const float *acc) {
  uint4 u;
  uint32_t *w = (uint32_t *)&u;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
    w[i] = *(const uint32_t *)&h;
  }
  return u;
}

__global__ void __launch_bounds__(256) embFwdKernel(const int64_t *tokens, const bf16 *wte, const bf16 *wpe, bf16 *x, int M, int T, int C, int V) {
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5), nv = C / 8;
  if (row >= M) return;
  const int64_t t = tokens[row];
  assert(t >= 0 && t < V);  // as the library's embedding has it
  const uint4 *a = (const uint4 *)(wte + (size_t)t * C), *b = (const uint4 *)(wpe + (size_t)(row % T) * C);
  uint4 *o = (uint4 *)(x + (size_t)row * C);
#pragma unroll 4
  for (int v = lane; v < nv; v += 32) {
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    addRow(s, a[v]);
    addRow(s, b[v]);
    o[v] = packRow(s);
  }
}

// MAXV: 256-column vectors per row that the registers are sized for.
template <int MAXV>
__global__ void __launch_bounds__(WARPS * 32, 1) embBwdKernel(const bf16 *dx, const int64_t *tokens, bf16 *dwte, bf16 *dwpe, int M, int T, int C,
                                                              int V) {
  extern __shared__ __align__(16) uint8_t embSmem[];
  __shared__ int heavy[HEAVY_LIST], nHeavy, paired[3], nPaired;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nv = C / 256;
  float *partial = (float *)embSmem;                // [WARPS][C]
  int *tok = (int *)(partial + (size_t)WARPS * C);  // [M, rounded up to 128]
  const int padded = (M + 127) / 128 * 128;
  if (threadIdx.x == 0) nHeavy = nPaired = 0;
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  if (dwte)
    for (int i = threadIdx.x; i < padded; i += WARPS * 32) {
      const int64_t t = i < M ? tokens[i] : -1;
      tok[i] = t >= 0 && t < V ? (int)t : -1;
    }
  __syncthreads();

  float acc[MAXV][8];
  auto clear = [&] {
#pragma unroll
    for (int v = 0; v < MAXV; v++)
#pragma unroll
      for (int k = 0; k < 8; k++) acc[v][k] = 0.f;
  };
  auto take = [&](int row) {
    uint4 r[MAXV];
    const uint4 *src = (const uint4 *)(dx + (size_t)row * C);
#pragma unroll
    for (int v = 0; v < MAXV; v++)
      if (v < nv) r[v] = src[v * 32 + lane];
#pragma unroll
    for (int v = 0; v < MAXV; v++)
      if (v < nv) addRow(acc[v], r[v]);
  };
  auto addInto = [&](bf16 *base, int row) {
    uint4 *dst = (uint4 *)(base + (size_t)row * C);
#pragma unroll
    for (int v = 0; v < MAXV; v++)
      if (v < nv) {
        addRow(acc[v], dst[v * 32 + lane]);
        dst[v * 32 + lane] = packRow(acc[v]);
      }
  };
  // which of the four tokens at base + 4 * lane are t and lie in [from, to)
  auto matches = [&](int base, int t, int from, int to) {
    const int4 q = *(const int4 *)(tok + base + 4 * lane);
    const int j = base + 4 * lane;
    unsigned m = (q.x == t ? 1u : 0u) | (q.y == t ? 2u : 0u) | (q.z == t ? 4u : 0u) | (q.w == t ? 8u : 0u);
    if (j < from) m &= from - j >= 4 ? 0u : 15u << (from - j);
    if (j + 4 > to) m &= to <= j ? 0u : 15u >> (j + 4 - to);
    return m;
  };
  // all rows of token t in [from, to), in order
  auto collect = [&](int t, int from, int to) {
    for (int base = from & ~127; base < to; base += 128) {
      const unsigned m = matches(base, t, from, to);
      for (unsigned any = __ballot_sync(0xffffffffu, m != 0); any; any &= any - 1) {
        const int l = __ffs(any) - 1;
        const unsigned ml = __shfl_sync(0xffffffffu, m, l);
#pragma unroll 1
        for (int c = 0; c < 4; c++)
          if (ml >> c & 1u) take(base + 4 * l + c);
      }
    }
  };

  if (dwte) {
    for (int k = warp; k * (int)gridDim.x + (int)blockIdx.x < M; k += WARPS) {
      const int i = k * gridDim.x + blockIdx.x, t = tok[i];
      if (t < 0) continue;
      bool first = true;
      for (int base = 0; base < i && first; base += 128) first = !__any_sync(0xffffffffu, matches(base, t, 0, i) != 0);
      if (!first) continue;
      int n = 0;
      for (int base = i & ~127; base < M; base += 128) n += __popc(matches(base, t, i, M));
      n = __reduce_add_sync(0xffffffffu, n);
      if (n > PAIRED && n > M / 4) {
        if (lane == 0) paired[atomicAdd(&nPaired, 1)] = i;
        continue;
      }
      if (n > HEAVY) {
        int at = 0;
        if (lane == 0) at = atomicAdd(&nHeavy, 1);
        at = __shfl_sync(0xffffffffu, at, 0);
        if (at < HEAVY_LIST) {
          if (lane == 0) heavy[at] = i;
          continue;
        }
      }
      clear();
      if (n == 1) take(i);
      else collect(t, i, M);
      addInto(dwte, t);
    }
  }
  if (dwpe) {
    for (int r = warp * gridDim.x + blockIdx.x; r < T; r += WARPS * gridDim.x) {
      clear();
#pragma unroll 2
      for (int row = r; row < M; row += T) take(row);
      addInto(dwpe, r);
    }
  }
  auto leave = [&](int w) {
    float *mine = partial + (size_t)w * C;
#pragma unroll
    for (int v = 0; v < MAXV; v++)
      if (v < nv) {
        float4 *d = (float4 *)(mine + (v * 32 + lane) * 8);
        d[0] = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
        d[1] = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
      }
  };
  __syncthreads();
  const int todo = min(nHeavy, HEAVY_LIST);
  for (int h = 0; h < todo; h++) {
    const int i = heavy[h], t = tok[i];
    const int per = (M - i + WARPS - 1) / WARPS, from = min(M, i + warp * per), to = min(M, from + per);
    clear();
    collect(t, from, to);
    leave(warp);
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += WARPS * 32) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; w++) s += partial[(size_t)w * C + c];
      bf16 *dst = dwte + (size_t)t * C + c;
      *dst = __float2bfloat16_rn(__bfloat162float(*dst) + s);
    }
    __syncthreads();
  }
  if (M <= PAIRED) return;  // launched without clusters
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int rank = (int)cluster.block_rank();
  for (int r = 0; r < 2; r++) {
    const int many = *cluster.map_shared_rank(&nPaired, r);
    for (int h = 0; h < many; h++) {
      const int i = *cluster.map_shared_rank(&paired[h], r), t = tok[i];
      clear();
      const int turn = rank * WARPS + warp;  // of 32 warps
      for (int base = i & ~31; base < M; base += 1024) {
        const int j = base + turn + 32 * lane;
        for (unsigned any = __ballot_sync(0xffffffffu, j >= i && j < M && tok[j] == t); any; any &= any - 1) take(base + turn + 32 * (__ffs(any) - 1));
      }
      leave(warp);
      cluster.sync();
      for (int c = rank * (C / 2) + threadIdx.x; c < (rank + 1) * (C / 2); c += WARPS * 32) {  // half of the columns each
        float s = 0.f;
        for (int q = 0; q < 2; q++) {
          const float *part = cluster.map_shared_rank(partial, q) + c;
#pragma unroll
          for (int w = 0; w < WARPS; w++) s += part[(size_t)w * C];
        }
        bf16 *dst = dwte + (size_t)t * C + c;
        *dst = __float2bfloat16_rn(__bfloat162float(*dst) + s);
      }
      cluster.sync();
    }
  }
  cluster.sync();  // nobody's shared memory goes before it has been read
}

}  // namespace

extern "C" {

// Whether the kernels take these sizes: rows of whole 256-column vectors, and few enough tokens for the search above.
int fcxEmbeddingTakes(int64_t M, int64_t C) { return M > 0 && M <= EMB_MAX_TOKENS && C % 256 == 0 && C > 0 && C <= 2048; }

cudaError_t fcxEmbeddingFwd(const int64_t *tokens, const void *wte, const void *wpe, void *x, int M, int T, int C, int V, cudaStream_t s) {
  if (!fcxEmbeddingTakes(M, C) || T <= 0 || M % T) return cudaErrorInvalidValue;
  if (((uintptr_t)wte | (uintptr_t)wpe | (uintptr_t)x) & 15) return cudaErrorInvalidValue;
  return fcxpdl::launchPdl(embFwdKernel, (M + 7) / 8, 256, 0, s, tokens, (const bf16 *)wte, (const bf16 *)wpe, (bf16 *)x, M, T, C, V);
}

cudaError_t fcxEmbeddingBwd(const void *dx, const int64_t *tokens, void *dwte, void *dwpe, int M, int T, int C, int V, cudaStream_t s) {
  if (!fcxEmbeddingTakes(M, C) || T <= 0 || M % T) return cudaErrorInvalidValue;
  if (((uintptr_t)dx | (uintptr_t)dwte | (uintptr_t)dwpe) & 15) return cudaErrorInvalidValue;
  const size_t smem = (size_t)WARPS * C * 4 + (size_t)(M + 127) / 128 * 128 * 4;  // at most 128 + 64 KB
  int grid = std::min(fcxhost::smCount(), (M + WARPS - 1) / WARPS);  // M >= T
  if (M > PAIRED) grid &= ~1;
  auto run = [&](auto kernel, int which) {
    static fcxhost::OncePerDevice once[2];
    const cudaError_t e = once[which]([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
    if (e != cudaSuccess) return e;
    return fcxpdl::launchPdlAttr(kernel, grid, WARPS * 32, smem, dim3(M > PAIRED ? 2 : 0, 1, 1), s, (const bf16 *)dx, tokens, (bf16 *)dwte, (bf16 *)dwpe, M, T, C, V);
  };
  return C <= 1024 ? run(embBwdKernel<4>, 0) : run(embBwdKernel<8>, 1);
}

}  // extern "C"

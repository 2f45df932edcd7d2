// Expert-parallel mixture-of-experts: dispatch and combine without a host
// round trip (one or several experts per rank).
//
//   fcxMoeDispatch  one cooperative kernel: counts the tokens bound for every
//                   expert, exchanges the count matrix with all ranks through
//                   the symmetric heap, derives this rank's write offsets on
//                   every expert, pushes each token's hidden vector straight
//                   into the expert rank's input buffer over NVLink together
//                   with a (source rank, token, choice) record, and returns
//                   once every source has finished writing into this rank.
//                   The number of rows received stays on the device.
//   (expert MLP)    grouped tcgen05 GEMMs with device-resident row counts
//                   (moe_gemm_sm100.cu); the down projection's epilogue
//                   stores every output row directly into the combine buffer
//                   of the rank the token came from.
//   fcxMoeCombine   waits for every CTA of every expert to report, then
//                   out[t] = sum_k w[t,k] * returned[t,k].
//
// With the reference a MoE layer needs flagcxAlltoAllv twice, whose counts and
// displacements are host arrays (flagcx/include/flagcx.h:397-401): the router
// result has to be copied to the host and the stream synchronised before the
// dispatch can even be issued.
#include "../kernels/prims.cuh"

#include <algorithm>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "device_state.h"
#include "moe_sm100.h"
#include "pdl.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int THREADS = 512;

__global__ void __launch_bounds__(THREADS, 1) moeDispatchKernel(const FcxDevComm dc, const FcxMoeParams p) {
  cg::grid_group grid = cg::this_grid();
  const int n = dc.nranks, me = dc.rank, L = p.L, E = n * L, capL = p.cap / L;
  const bool talk = n > 1 || p.exchange;
  const int entries = p.T * p.K;
  __shared__ int warpTotals[THREADS / 32];
  volatile int *err = p.errFlag;

  // ---- phase 1: CTA e numbers, in token order, the entries routed to expert e.  Every warp counts a contiguous stretch
  // of the entries, one barrier shares the counts, and a second look (in L1 by then) hands out the numbers.  In steps of
  // a whole CTA, four barriers each, 16384 entries took 32 dependent steps.
  if ((int)blockIdx.x < E) {
    const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int WARPS = THREADS / 32;
    const int per = ((entries + WARPS - 1) / WARPS + 31) / 32 * 32;
    const int lo = min(entries, warp * per), hi = min(entries, lo + per);
    int mine = 0;
#pragma unroll 8
    for (int i = lo + lane; i < hi; i += 32) mine += p.topkIdx[i] == e ? 1 : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) warpTotals[warp] = mine;
    __syncthreads();
    int running = 0, total = 0;
    for (int w = 0; w < WARPS; w++) {
      if (w < warp) running += warpTotals[w];
      total += warpTotals[w];
    }
#pragma unroll 4
    for (int base = lo; base < hi; base += 32) {
      const int i = base + lane;
      const bool hit = i < hi && p.topkIdx[i] == e;
      const unsigned ballot = __ballot_sync(0xffffffffu, hit);
      if (hit) p.slot[i] = running + __popc(ballot & ((1u << lane) - 1));
      running += __popc(ballot);
    }
    if (threadIdx.x == 0) p.localCounts[e] = total;
  }
  __threadfence();
  grid.sync();

  // ---- phase 2: every rank learns the whole count matrix [source][expert].  One rank alone has it already: no message, no
  // flag to wait for, and at the end nobody to tell, unless the caller asks for it all the same.
  if (talk && blockIdx.x == 0 && (int)threadIdx.x < n) {
    const int r = threadIdx.x;
    int *mat = (int *)(dc.heap[r] + p.countMatOff) + me * E;
    for (int e = 0; e < E; e++) mat[e] = p.localCounts[e];
    __threadfence_system();
    fcxdev::stRelease((uint64_t *)(dc.heap[r] + p.countFlagOff) + me, p.epoch);
  }
  __shared__ int baseOf[64];  // where this rank's tokens start in expert e's segment
  {
    bool ok = true;
    if (talk && (int)threadIdx.x < n)
      ok = fcxdev::waitGe(dc, (const uint64_t *)(dc.heap[me] + p.countFlagOff) + threadIdx.x, p.epoch, threadIdx.x, FCX_WAIT_DEVAPI,
                          blockIdx.x, p.epoch);
    if (!__syncthreads_and(ok)) { if (threadIdx.x == 0) *err = 1; }
    const int *mat = talk ? (const int *)(dc.heap[me] + p.countMatOff) : p.localCounts;
    if ((int)threadIdx.x < E) {
      int b = 0, tot = 0;
      for (int r = 0; r < n; r++) {
        int c = mat[r * E + threadIdx.x];
        if (r < me) b += c;
        tot += c;
      }
      baseOf[threadIdx.x] = b;
      if (tot > capL && blockIdx.x == 0) *err = 2;  // an expert's segment would overflow: tokens beyond the capacity are dropped
      if (!talk && blockIdx.x == 0) p.recvTotal[threadIdx.x] = min(tot, capL);
    }
    __syncthreads();
  }

  // ---- phase 3: one warp per (token, choice): push the hidden vector and its return address
  {
    const int warpsPerGrid = gridDim.x * (THREADS / 32);
    const int gw = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int vecs = p.H / 8;  // 16-byte vectors per token
    for (int i = gw; i < entries; i += warpsPerGrid) {
      const int e = p.topkIdx[i];
      if (e < 0 || e >= E) continue;
      const int inSeg = baseOf[e] + p.slot[i];
      if (inSeg >= capL) continue;
      const int dstRank = e / L, pos = (e % L) * capL + inSeg;
      const int t = i / p.K, k = i % p.K;
      const uint4 *src = (const uint4 *)((const __nv_bfloat16 *)p.x + (size_t)t * p.H);
      uint4 *dst = (uint4 *)(dc.heap[dstRank] + p.recvOff + (size_t)pos * p.H * 2);
      int v = lane;
      for (; v + 224 < vecs; v += 256) {  // eight 16-byte loads in flight per lane
        uint4 r[8];
#pragma unroll
        for (int j = 0; j < 8; j++) r[j] = src[v + 32 * j];
#pragma unroll
        for (int j = 0; j < 8; j++) dst[v + 32 * j] = r[j];
      }
      for (; v + 96 < vecs; v += 128) {
        uint4 a = src[v], b = src[v + 32], c = src[v + 64], d = src[v + 96];
        dst[v] = a; dst[v + 32] = b; dst[v + 64] = c; dst[v + 96] = d;
      }
      for (; v < vecs; v += 32) dst[v] = src[v];
      if (lane == 0) ((int4 *)(dc.heap[dstRank] + p.infoOff))[pos] = make_int4(me, t, k, 0);
    }
  }
  if (!talk) return;
  __threadfence_system();
  grid.sync();

  // ---- phase 4: tell every expert that this source is done; wait for all sources of this expert
  if (blockIdx.x == 0) {
    if ((int)threadIdx.x < n) fcxdev::stRelease((uint64_t *)(dc.heap[threadIdx.x] + p.doneOff) + me, p.epoch);
    bool ok = true;
    if ((int)threadIdx.x < n)
      ok = fcxdev::waitGe(dc, (const uint64_t *)(dc.heap[me] + p.doneOff) + threadIdx.x, p.epoch, threadIdx.x, FCX_WAIT_DEVAPI, 0, p.epoch);
    if (!__syncthreads_and(ok)) { if (threadIdx.x == 0) *err = 1; }
    if ((int)threadIdx.x < L) {
      const int *mat = (const int *)(dc.heap[me] + p.countMatOff);
      int tot = 0;
      for (int r = 0; r < n; r++) tot += mat[r * E + me * L + threadIdx.x];
      p.recvTotal[threadIdx.x] = min(tot, capL);
    }
  }
}

// The dispatch of one rank that exchanges nothing (p.exchange 0): no cooperative launch, no barrier of the grid and nobody to
// wait for.  Every CTA numbers its own stretch of the entries after counting, by itself, the entries before it per expert
// (in registers, eight experts to a 64-bit word), so the only order between CTAs is that of the launches around it.  The
// first row of every warp is already on its way while it counts.  The numbers are those of the cooperative kernel (token
// order within an expert).  Bound by latency on small batches and by memory on large ones, where 32 warps per SM keep 128 KB of
// rows in flight.  On 64 SMs, cooperative kernel / this one, us: 512 tokens x 1024 with two choices of 4 experts 7.6 / 3.7, 2048 x
// 2048 (8 experts) 13.9 / 9.6, 8192 x 4096 64.5 / 51.2; on 148 SMs 7.8 / 3.7, 10.8 / 7.1, 45.1 / 37.8.
//
// The counting is every CTA's own, so the grid's reads of the entries grow with CTAs x entries x experts / 8.  The bounds on
// CTAs (the SMs that the caller allows) and on a CTA's entries keep that below what the barriers of the cooperative kernel cost, up to
// the largest sizes they admit: 131072 entries of 64 experts on 148 SMs 96 us, 122 there (with rows of 64), 111 / 192 (of 512).
constexpr int LOCAL_CHUNK = 1024;  // most entries of one CTA
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) moeDispatchLocalKernel(const FcxDevComm dc, const FcxMoeParams p) {
  const int E = p.L, capL = p.cap / p.L, entries = p.T * p.K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int WARPS = NT / 32;
  __shared__ int count[64], slotOf[LOCAL_CHUNK], expertOf[LOCAL_CHUNK];
  const int per = (entries + gridDim.x - 1) / gridDim.x;
  const int lo = (int)min((long long)entries, (long long)blockIdx.x * per), hi = min(entries, lo + per);
  if (threadIdx.x < 64) count[threadIdx.x] = 0;
  fcxpdl::pdlWait();
  fcxpdl::pdlRelease();  // what comes next may rely on everything before this kernel, too
  const int vecs = p.H / 8;  // 16-byte vectors per token
  uint4 head[8];             // the first 256 vectors of this warp's first row
  auto rowOf = [&](int i) { return (const uint4 *)((const __nv_bfloat16 *)p.x + (size_t)(i / p.K) * p.H); };
  if (lo + warp < hi) {
    const uint4 *src = rowOf(lo + warp);
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (lane + 32 * j < vecs) head[j] = src[lane + 32 * j];
  }
  for (int i = lo + threadIdx.x; i < hi; i += NT) expertOf[i - lo] = p.topkIdx[i];
  __syncthreads();
  for (int e0 = 0; e0 < E; e0 += 8) {
    // at most 128 entries of a thread between two turns of the outer loop: a byte per expert holds them
    for (int from = 0; from < lo; from += 128 * NT) {
      const int to = min(lo, from + 128 * NT);
      uint64_t c = 0;
#pragma unroll 8
      for (int i = from + (int)threadIdx.x; i < to; i += NT) {
        const uint32_t d = (uint32_t)(p.topkIdx[i] - e0);
        c += d < 8u ? 1ull << (8 * d) : 0ull;
      }
      for (int d = 0; d < 8 && e0 + d < E; d++) {
        const uint32_t sum = __reduce_add_sync(0xffffffffu, (uint32_t)(c >> (8 * d)) & 255u);
        if (lane == 0 && sum) atomicAdd(&count[e0 + d], (int)sum);
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    for (int base = lo; base < hi; base += 32) {
      const bool in = base + lane < hi;
      const int e = in ? expertOf[base + lane - lo] : -1;
      const bool good = e >= 0 && e < E;
      const unsigned same = __match_any_sync(0xffffffffu, good ? e : -1);
      const int at = good ? count[e] + __popc(same & ((1u << lane) - 1)) : 0;
      __syncwarp();
      if (good && (same >> lane) == 1u) count[e] = at + 1;  // the last lane of its expert
      if (in) {
        slotOf[base + lane - lo] = at;
        p.slot[base + lane] = at;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  if (blockIdx.x == gridDim.x - 1 && (int)threadIdx.x < E) {  // the last stretch ends with the last entry: these are the totals
    const int tot = count[threadIdx.x];
    p.localCounts[threadIdx.x] = tot;
    p.recvTotal[threadIdx.x] = min(tot, capL);
    if (tot > capL) *(volatile int *)p.errFlag = 2;  // an expert's segment would overflow: entries beyond the capacity are dropped
  }
  for (int i = lo + warp; i < hi; i += WARPS) {
    const int e = expertOf[i - lo], inSeg = slotOf[i - lo];
    if (e < 0 || e >= E || inSeg >= capL) continue;
    const int pos = e * capL + inSeg;
    const uint4 *src = rowOf(i);
    uint4 *dst = (uint4 *)(dc.heap[dc.rank] + p.recvOff + (size_t)pos * p.H * 2);
    if (lane == 0) ((int4 *)(dc.heap[dc.rank] + p.infoOff))[pos] = make_int4(dc.rank, i / p.K, i % p.K, 0);
    for (int v = 0; v < vecs; v += 256) {
      if (i != lo + warp || v > 0) {
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (v + lane + 32 * j < vecs) head[j] = src[v + lane + 32 * j];
      }
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (v + lane + 32 * j < vecs) dst[v + lane + 32 * j] = head[j];
    }
  }
}

// h[r, f] = silu(g[r, f]) * u[r, f] with gu = [g | u] of width 2F; rows beyond *rows are skipped
__global__ void __launch_bounds__(256) siluMulKernel(const __nv_bfloat16 *__restrict__ gu, __nv_bfloat16 *__restrict__ h, const int *rows,
                                                     int maxRows, int F) {
  const int R = rows ? min(*rows, maxRows) : maxRows;
  const size_t vecPerRow = F / 8, total = (size_t)R * vecPerRow;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t r = i / vecPerRow, c = i % vecPerRow;
    uint4 gv = *(const uint4 *)(gu + r * 2 * F + c * 8), uv = *(const uint4 *)(gu + r * 2 * F + F + c * 8);
    const __nv_bfloat162 *g2 = (const __nv_bfloat162 *)&gv, *u2 = (const __nv_bfloat162 *)&uv;
    uint4 o;
    __nv_bfloat162 *o2 = (__nv_bfloat162 *)&o;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float2 g = __bfloat1622float2(g2[j]), u = __bfloat1622float2(u2[j]);
      float a = g.x / (1.f + __expf(-g.x)) * u.x, b = g.y / (1.f + __expf(-g.y)) * u.y;
      o2[j] = __floats2bfloat162_rn(a, b);
    }
    *(uint4 *)(h + r * F + c * 8) = o;
  }
}

// out[t] = sum_k w[t,k] * ret[t,k], after every CTA of every expert's output GEMM has reported.
// KC > 0: K is KC (1 to 4), 8 / KC output vectors per thread and step with every choice's row loaded before the first is
// used, eight 16-byte loads in flight (six for three choices); positions in 32 bits (their 64-bit divisions cost more than the
// loads).  Three choices took 70 us one vector at a time and take 51 so at 8192 x 4096; two take 36, four 55.
// KC = 0: any K and any size, one vector at a time.
template <int KC>
__global__ void __launch_bounds__(256) moeCombineKernel(const FcxDevComm dc, const __nv_bfloat16 *ret, const float *w, __nv_bfloat16 *out, int T,
                                                        int H, int K, size_t doneOff, uint64_t want, int *errFlag) {
  bool ok = true;
  fcxpdl::pdlWait();
  if (threadIdx.x == 0) {
    ok = fcxdev::waitGe(dc, (const uint64_t *)(dc.heap[dc.rank] + doneOff), want, -1, FCX_WAIT_DEVAPI, blockIdx.x, want);
    if (!ok) *errFlag = 1;
  }
  if (!__syncthreads_and(ok)) return;
  const size_t vecPerRow = H / 8, total = (size_t)T * vecPerRow, stride = (size_t)gridDim.x * blockDim.x;
  if constexpr (KC > 0) {
    constexpr int U = 8 / KC;
    const uint32_t tot = (uint32_t)total, per = (uint32_t)vecPerRow, step = (uint32_t)stride;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < tot; i += U * step) {
      uint4 v[U][KC];
      float wk[U][KC];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const uint32_t pos = min(i + u * step, tot - 1), t = pos / per, c = pos - t * per;
#pragma unroll
        for (int k = 0; k < KC; k++) {
          wk[u][k] = w[t * KC + k];
          // volatile: the compiler would move each load behind the test of its weight, one at a time
          asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(v[u][k].x), "=r"(v[u][k].y), "=r"(v[u][k].z), "=r"(v[u][k].w)
                       : "l"(ret + ((size_t)t * KC + k) * H + c * 8) : "memory");
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < KC; k++) {
          // a choice that was not dispatched (expert id out of range, capacity overflow) has weight 0 and whatever the
          // buffer holds in the place of a row
          if (wk[u][k] == 0.f) v[u][k] = make_uint4(0, 0, 0, 0);
          const __nv_bfloat162 *h2 = (const __nv_bfloat162 *)&v[u][k];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float2 f = __bfloat1622float2(h2[j]);
            acc[2 * j] += wk[u][k] * f.x;
            acc[2 * j + 1] += wk[u][k] * f.y;
          }
        }
        uint4 o;
        __nv_bfloat162 *o2 = (__nv_bfloat162 *)&o;
#pragma unroll
        for (int j = 0; j < 4; j++) o2[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
        const uint32_t pos = i + u * step;
        if (pos < tot) *(uint4 *)(out + (size_t)pos * 8) = o;  // out is contiguous
      }
    }
  } else {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
      const size_t t = i / vecPerRow, c = i % vecPerRow;
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int k = 0; k < K; k++) {
        const float wk = w[t * K + k];
        if (wk == 0.f) continue;  // a choice that was not dispatched (expert id out of range, capacity overflow) has no row
        uint4 v = *(const uint4 *)(ret + ((t * K + k) * H) + c * 8);
        const __nv_bfloat162 *h2 = (const __nv_bfloat162 *)&v;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          float2 f = __bfloat1622float2(h2[j]);
          acc[2 * j] += wk * f.x;
          acc[2 * j + 1] += wk * f.y;
        }
      }
      uint4 o;
      __nv_bfloat162 *o2 = (__nv_bfloat162 *)&o;
#pragma unroll
      for (int j = 0; j < 4; j++) o2[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
      *(uint4 *)(out + t * H + c * 8) = o;
    }
  }
}

}  // namespace

// The launch of a dispatch that exchanges nothing: CTAs of moeDispatchLocalKernel (and `threads` of each), or 0 for the cooperative
// kernel.  `ctas` is the number of SMs that the caller lets the dispatch have, so no more CTAs than that are launched; where their
// shared memory does not hold the entries, the cooperative kernel has as many CTAs.  A CTA has 16 warps up to eight entries for
// each (less set-up), 32 beyond (more rows in flight).  16 / 32 warps, us: 4096 entries x 2048 on 148 SMs (1.7 entries per warp of 16)
// 7.1 / 7.4, on 64 (4) 9.6 / 9.9, 16384 x 4096 on 148 (7) 37.8 / 40.1, on 64 (16) 56.1 / 51.2, 32768 x 1024 on 148 (14) 23.7 / 20.3.
extern "C" int fcxMoeDispatchPlan(int64_t entries, int ctas, int sms, int *threads) {
  const int64_t most = std::max(1, std::min(ctas, sms));
  *threads = entries <= 8 * 16 * most ? 512 : 1024;
  const int64_t warps = *threads / 32, grid = std::max<int64_t>(1, std::min(most, (entries + warps - 1) / warps));
  if ((entries + grid - 1) / grid > LOCAL_CHUNK) return 0;
  return (int)grid;
}

extern "C" cudaError_t fcxMoeDispatch(const FcxDevComm *dc, const FcxMoeParams *p, int ctas, cudaStream_t s) {
  if (p->H % 8 || p->K < 1 || dc->nranks > FCX_MAX_RANKS || p->L < 1 || dc->nranks * p->L > 64 || p->cap % p->L) return cudaErrorInvalidValue;
  const int sms = fcxhost::smCount();
  if (dc->nranks == 1 && !p->exchange) {
    int threads = 0;
    const int grid = fcxMoeDispatchPlan((int64_t)p->T * p->K, ctas, sms, &threads);
    if (grid) return fcxpdl::launchPdl(threads == 512 ? moeDispatchLocalKernel<512> : moeDispatchLocalKernel<1024>, grid, threads, 0, s, *dc, *p);
  }
  ctas = std::max(dc->nranks * p->L, std::min(ctas, sms));  // one CTA per expert at least; all resident: the kernel synchronises the grid
  void *args[] = {(void *)dc, (void *)p};
  return cudaLaunchCooperativeKernel((const void *)moeDispatchKernel, dim3(ctas), dim3(THREADS), args, 0, s);
}

extern "C" cudaError_t fcxSiluMul(const void *gu, void *h, const int *rows, int maxRows, int F, cudaStream_t s) {
  if (F % 8) return cudaErrorInvalidValue;
  siluMulKernel<<<592, 256, 0, s>>>((const __nv_bfloat16 *)gu, (__nv_bfloat16 *)h, rows, maxRows, F);
  return cudaGetLastError();
}

extern "C" cudaError_t fcxMoeCombine(const FcxDevComm *dc, const void *ret, const float *w, void *out, int T, int H, int K, size_t doneOff,
                                     uint64_t want, int *errFlag, cudaStream_t s) {
  if (H % 8) return cudaErrorInvalidValue;
  // positions may run past the total by up to eight grid strides
  const bool small = (uint64_t)T * (H / 8) + 16ull * 592 * 256 < (1ull << 32);
  auto kernel = !small ? moeCombineKernel<0> : K == 1 ? moeCombineKernel<1> : K == 2 ? moeCombineKernel<2> : K == 3 ? moeCombineKernel<3>
                : K == 4 ? moeCombineKernel<4> : moeCombineKernel<0>;
  return fcxpdl::launchPdl(kernel, 592, 256, 0, s, *dc, (const __nv_bfloat16 *)ret, w, (__nv_bfloat16 *)out, T, H, K, doneOff, want, errFlag);
}

// The low-latency reductions (all-reduce, reduce-scatter and reduce of at most 32 KB) as kernels of their own.
//
// Such a call is a handful of trips to memory, so what surrounds them counts: inside the kernel that holds every staged
// collective these few instructions were spread over a large body, and each launch had to fetch it anew.
// The kernel of an all-reduce of 4 KB, in us before that and the opening in one trip (prims.cuh) and with both: 8 emulated
// ranks 10.6 -> 9.3, 2 ranks 8.4 -> 7.0; reduce-scatter of 2 KB pieces among 8 10.9 -> 9.1.
#include "lowlatency.cuh"
#include "launch.h"
#include "dispatch.h"

#include <cuda_runtime.h>

namespace fcxdev {

// The pair of lines of a peer's unit is looked at once more for the report: the tag of an earlier collective tells a peer that
// is behind from one that never wrote.  Kept out of the wait itself, which it would slow down.
static __device__ __noinline__ void giveUpOnLine(const FcxDevComm &dc, uint32_t code, int peer, size_t llOff, size_t u, int cta, uint32_t tag,
                                                 uint64_t seq) {
  const char *line = dc.heap[dc.rank] + llOff + (size_t)peer * FCX_LL_SLOT_BYTES + u * 32;
  const uint32_t first = llLoad(line).y, second = llLoad(line + 16).y;
  giveUp(dc, code, peer, FCX_WAIT_LL, cta, tag, first != tag ? first : second, seq);
}

// mode 0: all-reduce (everybody sends its whole vector to everybody and reduces);
// mode 1: reduce-scatter (piece p goes to rank p, every rank reduces the pieces it received and its own);
// mode 2: reduce (everybody sends its whole vector to the root, which reduces).
template <typename T>
__device__ void arLL(const FcxDevComm &dc, const FcxCollArgs &a, uint64_t seq, int cta, int nctas, int mode = 0) {
  using Acc = typename Elem<T>::Acc;
  constexpr int G = 16 / (int)sizeof(T);
  const int n = dc.nranks, me = dc.rank;
  const uint32_t tag = (uint32_t)seq;
  const size_t gtid = (size_t)cta * blockDim.x + threadIdx.x, gstride = (size_t)nctas * blockDim.x;
  const size_t nunits = (a.count + G - 1) / G;
  const size_t pieceBytes = mode == 1 ? a.sendStride * sizeof(T) : 0;  // distance between the pieces of a reduce-scatter
  const char *send = (const char *)a.send + (size_t)me * pieceBytes;    // what this rank contributes to its own result
  const bool reduces = mode != 2 || me == a.root;
  const bool alS = aligned16(send), alR = aligned16(a.recv);
  const size_t llOff = FCX_OFF_LL + (size_t)(seq & 1) * FCX_MAX_RANKS * FCX_LL_SLOT_BYTES;
  // All lines go out before any is waited for, and every peer's line of a unit is asked for before the first is used: a
  // line at a time, the kernel spent a trip to L2 per peer and unit one after the other (7 x 0.5 us with eight ranks).
  for (size_t u = gtid; u < nunits; u += gstride) {
    const int nv = (int)min((size_t)G, a.count - u * G);
    Acc mine[G];
    uint4 raw;
    if (mode != 1) {
      loadUnit<T, G>(send + u * 16, alS, nv, mine);
      packUnit<T, G>(mine, &raw);
    }
    for (int k = 1; k < n; k++) {
      int p = (me + k) % n;
      if (mode == 2 && p != a.root) continue;
      if (mode == 1) {
        const char *src = (const char *)a.send + (size_t)p * pieceBytes + u * 16;
        loadUnit<T, G>(src, aligned16(src), nv, mine);
        packUnit<T, G>(mine, &raw);
      }
      char *line = dc.heap[p] + llOff + (size_t)me * FCX_LL_SLOT_BYTES + u * 32;
      llStore(line, raw.x, raw.y, tag);
      llStore(line + 16, raw.z, raw.w, tag);
    }
  }
  if (!reduces) return;
  const char *lines = dc.heap[me] + llOff;
  for (size_t u = gtid; u < nunits; u += gstride) {
    const int nv = (int)min((size_t)G, a.count - u * G);
    Acc mine[G];
    loadUnit<T, G>(send + u * 16, alS, nv, mine);
    uint4 lo[FCX_MAX_RANKS], hi[FCX_MAX_RANKS];
    unsigned pending = ((1u << n) - 1u) & ~(1u << me), spins = 0;
    uint64_t t0 = 0;
    for (;;) {
#pragma unroll
      for (int p = 0; p < FCX_MAX_RANKS; p++)
        if (pending >> p & 1u) {
          lo[p] = llLoad(lines + (size_t)p * FCX_LL_SLOT_BYTES + u * 32);
          hi[p] = llLoad(lines + (size_t)p * FCX_LL_SLOT_BYTES + u * 32 + 16);
        }
#pragma unroll
      for (int p = 0; p < FCX_MAX_RANKS; p++)
        if ((pending >> p & 1u) && lo[p].y == tag && lo[p].w == tag && hi[p].y == tag && hi[p].w == tag) pending &= ~(1u << p);
      if (!pending) break;
      if (spins == 0) t0 = globalTimerNs();
      if ((++spins & 63u) == 0u) {
        const int late = __ffs(pending) - 1;
        if (*(volatile unsigned int *)&localOf(dc)->abortSeen) return;
        if (globalTimerNs() - t0 > dc.timeoutNs) {
          giveUpOnLine(dc, FCX_ERR_TIMEOUT, late, llOff, u, cta, tag, seq);
          return;
        }
        if ((spins & 1023u) == 0u && *dc.abortWord) {
          giveUpOnLine(dc, FCX_ERR_ABORT, late, llOff, u, cta, tag, seq);
          return;
        }
      }
    }
    Acc acc[G];
#pragma unroll
    for (int p = 0; p < FCX_MAX_RANKS; p++)  // in rank order on every rank
      if (p < n) {
        Acc in[G];
        if (p == me) {
#pragma unroll
          for (int i = 0; i < G; i++) in[i] = mine[i];
        } else {
          union { uint4 v; T t[G]; } w;
          w.v = make_uint4(lo[p].x, lo[p].z, hi[p].x, hi[p].z);
#pragma unroll
          for (int i = 0; i < G; i++) in[i] = Elem<T>::up(w.t[i]);
        }
#pragma unroll
        for (int i = 0; i < G; i++) acc[i] = p == 0 ? in[i] : applyOp<Acc>(acc[i], in[i], a.redop);
      }
#pragma unroll
    for (int i = 0; i < G; i++) acc[i] = finish<Acc>(acc[i], a.redop, n, a.scale);
    uint4 outv;
    packUnit<T, G>(acc, &outv);
    storeUnit<T, G>((char *)a.recv + u * 16, alR, nv, &outv);
  }
}

template <typename T>
__device__ __forceinline__ void fcxLlBody(const FcxDevComm &dc, const FcxCollArgs &a, int cta, int nctas) {
  uint64_t seq;
  if (!prologue(dc, cta, &seq)) return;
  if (a.count * sizeof(T) > FCX_LL_MAX_PAYLOAD) {
    if (threadIdx.x == 0) giveUp(dc, FCX_ERR_BADARG, dc.rank, FCX_WAIT_BARRIER, cta, dc.stageBytes, ~0ull, seq);
  } else {
    arLL<T>(dc, a, seq, cta, nctas, a.kind == FCX_K_RS_LL ? 1 : a.kind == FCX_K_REDUCE_LL ? 2 : 0);
  }
  epilogue(dc, seq, nctas);
}

template <typename T>
__global__ void __launch_bounds__(FCX_THREADS, 1) fcxLlKernel(FcxDevComm dc, FcxCollArgs a) {
  fcxLlBody<T>(dc, a, blockIdx.x, gridDim.x);
}
template <typename T>
__global__ void __launch_bounds__(FCX_THREADS, 1) fcxLlEmuKernel(const __grid_constant__ FcxEmuRanks l, int ctasPerRank) {
  __shared__ FcxDevComm dc;
  __shared__ FcxCollArgs a;
  emuRank(l, blockIdx.x / ctasPerRank, &dc, &a);
  fcxLlBody<T>(dc, a, blockIdx.x % ctasPerRank, ctasPerRank);
}

}  // namespace fcxdev

using namespace fcxdev;

namespace {

template <typename T>
cudaError_t launchLl(const FcxDevComm &dc, const FcxCollArgs &a, int nctas, cudaStream_t s) {
  fcxLlKernel<T><<<nctas, FCX_THREADS, 0, s>>>(dc, a);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launchLlEmu(const FcxEmuRanks &l, int nranks, int nctas, cudaStream_t s) {
  void *params[] = {(void *)&l, (void *)&nctas};
  return cudaLaunchCooperativeKernel((const void *)fcxLlEmuKernel<T>, dim3(nranks * nctas), dim3(FCX_THREADS), params, 0, s);
}

}  // namespace

extern "C" cudaError_t fcxLaunchLl(const FcxDevComm *dc, const FcxCollArgs *a, int nctas, cudaStream_t s) {
#define CALL(TI, TO) launchLl<TI>(*dc, *a, nctas, s)
  FCX_DISPATCH_SAME(a->dtype, CALL)
#undef CALL
}

extern "C" cudaError_t fcxLaunchLlEmu(const FcxEmuRanks *l, int nranks, int nctas, cudaStream_t s) {
#define CALL(TI, TO) launchLlEmu<TI>(*l, nranks, nctas, s)
  FCX_DISPATCH_SAME(l->args[0].dtype, CALL)
#undef CALL
}

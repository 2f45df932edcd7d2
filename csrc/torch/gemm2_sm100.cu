// bf16 GEMM on CTA pairs: tcgen05.mma.cta_group::2 (M 256, N 256, K 16 per instruction).
//
//   C[M,N] = A[M,K] * B[N,K]^T (+ bias), operands K-major or MN-major as in the one-CTA kernel.
//
// Two CTAs of a cluster, resident on the two SMs of one pair, work on one 256 x 256 output tile.  Each CTA
// loads ITS 128 rows of A and ITS 128 of the 256 columns of B into its own shared memory (plain TMA loads, never
// multicast); the instruction, issued by one thread of the pair's leader CTA, reads the A half of each CTA for that
// CTA's 128 accumulator rows and the two B halves for the 256 columns, and writes each CTA's accumulator into that
// CTA's own TMEM.  Against the one-CTA kernel (128 x 256 tile, 48 KB per K block of 64 through one SM's shared
// memory) a CTA now feeds 32 KB per K block for the same math, which lifts the shared-memory bound on the MMA rate
// and halves the L2 reads of B; the smaller stage also buys a 5-deep pipeline.
//
// Roles per CTA (384 threads): warp 0 TMA producer, warp 1 MMA issuer (leader CTA only), warp 2 TMEM allocation,
// warps 4-11 epilogue (TMEM -> registers -> bf16 blocks in shared memory -> TMA store, or TMA add for split K and
// accumulated gradients).
// Barriers: the leader's full[stage] collects the bytes of both CTAs' loads; tcgen05.commit arrives on empty[stage]
// and accFull[buf] of BOTH CTAs (barrier multicast inside the cluster; that is a signal, not a load); the epilogue
// warps of both CTAs arrive on the leader's accEmpty[buf].  Every wait is bounded: after the limit the kernel
// records an error, leaves its loops, meets its peer at the closing cluster barrier, frees its TMEM and returns.
//
// The reference has no GEMM; this kernel serves the model's projections (forward, input gradient, weight gradient).
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <vector>

#include "device_state.h"
#include "gemm_sm100.h"
#include "gemm_units.h"
#include "pdl.cuh"
#include "tcgen05.cuh"

namespace {

using namespace fcxmma;

constexpr int BM = 128;    // accumulator rows per CTA (256 per pair)
constexpr int BN = 256;    // columns per tile
constexpr int BNH = 128;   // B columns that one CTA holds
#ifndef FCX_PAIR_STAGES
#define FCX_PAIR_STAGES 5
#endif
constexpr int BK = 64, STAGES = FCX_PAIR_STAGES;
constexpr int STG_DEPTH = STAGES >= 6 ? 1 : 2;  // staging blocks per epilogue warp: the sixth stage takes the room of the second block
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BNH * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int STG_BYTES = 32 * 64;                 // staging block: 32 rows x 32 bf16 columns
constexpr int EPI_BYTES = 8 * STG_DEPTH * STG_BYTES;  // 8 epilogue warps
constexpr int BIAS_BYTES = 8 * 128 * 4;  // per epilogue warp: its 128 bias values as fp32
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + BIAS_BYTES + 1024 + 256;
constexpr int THREADS = 384;
constexpr int MN_BLOCK_BYTES = 64 * BK * 2;

// D fp32, A/B bf16, M = 256 over the pair, N = 256.
__device__ __forceinline__ uint32_t instrDescPair(int aMN, int bMN) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(aMN ? 1 : 0) << 15) | ((uint32_t)(bMN ? 1 : 0) << 16) |
         ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
}

// Tile t -> (256-row block, 256-column block); bands of `group` row blocks as in the one-CTA kernel.
__device__ __forceinline__ void tileCoord2(int group, int nM, int nN, int t, int *mb, int *nb) {
  if (group > 0) {
    const int perBand = group * nN, band = t / perBand, first = band * group;
    const int rowsHere = min(group, nM - first), within = t - band * perBand;
    *mb = first + within % rowsHere;
    *nb = within / rowsHere;
  } else {
    *mb = t / nN;
    *nb = t % nN;
  }
}

// tanh-form GELU, the same arithmetic as the stand-alone bias+GELU kernel of the training ops
__device__ __forceinline__ float geluTanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(k0 * (x + k1 * x * x * x)));
  return 0.5f * x * (1.f + t);
}

// What the kernel needs of one product; `units` counts its tiles times its K pieces.
struct PairProb {
  CUtensorMap a, b, c;
  int M, N, K, aMN, bMN, splitK, accumulate, group, units;
};
struct PairArgs {
  PairProb prob[2];
  CUtensorMap c2;  // GELU: the second output
  const void *bias;
  int extra;
  int *errFlag;
};

// MODE_PLAIN: one product.  MODE_GELU: two outputs per tile: C = A B^T (kept for the backward pass) and
// C2 = gelu(A B^T + bias).  MODE_DUAL: two independent products in one launch (the input and weight gradients of a linear
// layer), so that the units of one fill the last wave of the other.
enum { MODE_PLAIN, MODE_GELU, MODE_DUAL };
template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    fcxGemmPairKernel(const __grid_constant__ PairArgs args) {
  extern __shared__ uint8_t smemRaw[];
  const int warp = warpIndex(), lane = threadIdx.x & 31;
  volatile int *err = args.errFlag;
  const uint32_t cr = ctaRankInCluster();  // 0 = leader
  const int pair = blockIdx.x >> 1, nPairs = gridDim.x >> 1;

  uint8_t *tiles = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t *epiStage = tiles + STAGES * STAGE_BYTES;
  float *biasStage = (float *)(epiStage + EPI_BYTES);
  uint64_t *bars = (uint64_t *)(epiStage + EPI_BYTES + BIAS_BYTES);
  uint64_t *fullBar = bars, *emptyBar = bars + STAGES, *accFull = bars + 2 * STAGES, *accEmpty = bars + 2 * STAGES + 2;
  uint32_t *tmemBaseSlot = (uint32_t *)(bars + 2 * STAGES + 4);

  // Unit u of a product -> its tile and K range.
  struct Where {
    int mb, nb, kLo, kHi;
    bool first;
  };
  auto locate = [](const PairProb &p, int u) {
    Where w;
    const int nN = (p.N + BN - 1) / BN, nM = (p.M + 2 * BM - 1) / (2 * BM), nK = (p.K + BK - 1) / BK;
    const int kPer = (nK + p.splitK - 1) / p.splitK, piece = u % p.splitK;
    tileCoord2(p.group, nM, nN, u / p.splitK, &w.mb, &w.nb);
    w.kLo = piece * kPer;
    w.kHi = min(nK, w.kLo + kPer);
    w.first = piece == 0;
    return w;
  };
  UnitIter it(pair, nPairs, args.prob[0].units, MODE == MODE_DUAL ? args.prob[1].units : 0, args.extra);
  int which, unit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbarInit(&fullBar[s], 1); mbarInit(&emptyBar[s], 1); }
    for (int b = 0; b < 2; b++) { mbarInit(&accFull[b], 1); mbarInit(&accEmpty[b], 16); }  // 8 epilogue warps in each CTA
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemBaseSlot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fenceBefore();
  __syncthreads();
  clusterSync();  // the peer's barriers exist before anything arrives on them
  fenceAfter();
  const uint32_t tmemBase = *tmemBaseSlot;
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();  // everything above touches only this CTA's own memories

  if (warp == 0) {
    // ---- TMA producer (both CTAs): own half of A and of B; bytes counted on the leader's barrier
    if (electOne()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      while (ok && it.next(&which, &unit)) {
        const PairProb &p = args.prob[MODE == MODE_DUAL ? which : 0];
        const Where w = locate(p, unit);
        const int rowA = w.mb * 2 * BM + (int)cr * BM, colB = w.nb * BN + (int)cr * BNH;
        for (int kb = w.kLo; kb < w.kHi; kb++) {
          if (!mbarWait(&emptyBar[stage], phase ^ 1, err)) { ok = false; break; }
          if (cr == 0) mbarExpectTx(&fullBar[stage], 2 * STAGE_BYTES);
          const uint32_t bar = mapToCta(smemAddr(&fullBar[stage]), 0);
          uint8_t *sa = tiles + stage * STAGE_BYTES, *sb = sa + A_BYTES;
          if (p.aMN) {
            for (int j = 0; j < BM / 64; j++) tmaLoad2dPair(sa + j * MN_BLOCK_BYTES, &p.a, rowA + j * 64, kb * BK, bar);
          } else {
            tmaLoad2dPair(sa, &p.a, kb * BK, rowA, bar);
          }
          if (p.bMN) {
            for (int j = 0; j < BNH / 64; j++) tmaLoad2dPair(sb + j * MN_BLOCK_BYTES, &p.b, colB + j * 64, kb * BK, bar);
          } else {
            tmaLoad2dPair(sb, &p.b, kb * BK, colB, bar);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one thread of the leader CTA drives the tensor cores of both SMs; the warp waits as one
    if (cr == 0) {
      int stage = 0, buf = 0;
      uint32_t phase = 0, accPhase = 0;
      bool ok = true;
      while (ok && it.next(&which, &unit)) {
        const PairProb &p = args.prob[MODE == MODE_DUAL ? which : 0];
        const Where w = locate(p, unit);
        const bool aMN = p.aMN, bMN = p.bMN;
        const uint32_t idesc = instrDescPair(aMN, bMN);
        if (!__all_sync(0xffffffffu, mbarWait(&accEmpty[buf], accPhase ^ 1, err))) break;
        fenceAfter();
        const uint32_t dTmem = tmemBase + (uint32_t)buf * BN;
        for (int kb = w.kLo; kb < w.kHi; kb++) {
          if (!__all_sync(0xffffffffu, mbarWait(&fullBar[stage], phase, err))) { ok = false; break; }
          fenceAfter();
          if (electOne()) {
            const uint32_t sa = smemAddr(tiles + stage * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / 16; k++) {
              const uint64_t da = aMN ? smemDescMN(sa + k * 2048, MN_BLOCK_BYTES) : smemDesc(sa + k * 32);
              const uint64_t db = bMN ? smemDescMN(sb + k * 2048, MN_BLOCK_BYTES) : smemDesc(sb + k * 32);
              mmaF16Pair(dTmem, da, db, idesc, (kb > w.kLo || k > 0) ? 1u : 0u);
            }
            mmaCommitPair(&emptyBar[stage]);
            if (kb + 1 == w.kHi) mmaCommitPair(&accFull[buf]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (++buf == 2) { buf = 0; accPhase ^= 1; }
      }
    }
  } else if (warp >= 4) {
    // ---- epilogue (both CTAs, 8 warps): warp w owns TMEM lanes [32*(w%4), +32) = 32 of this CTA's 128 rows, and the
    // left (warps 4-7) or right (warps 8-11) 128 of the tile's 256 columns.  32 columns at a time: tcgen05.ld (one row
    // per lane), bias, fp32 -> bf16, 16-byte stores into a staging block laid out as the TMA's 64-byte swizzle wants it
    // (conflict-free), then ONE thread hands the 32 x 32 block to the TMA unit, as a store or, for a piece of a split K
    // or an accumulated gradient, as a reduction (add) into C.  The TMA clips what lies beyond M and N.  Two staging
    // blocks per warp: the next block is filled while the unit still reads the previous one.
    const int ew = warp - 4, q = ew & 3, half = ew >> 2;
    int buf = 0;
    uint32_t accPhase = 0, chunkNo = 0;
    bool live = true;
    uint8_t *stgBase = epiStage + (size_t)ew * STG_DEPTH * STG_BYTES;
    float *biasW = biasStage + ew * 128;
    while (it.next(&which, &unit)) {
      const PairProb &p = args.prob[MODE == MODE_DUAL ? which : 0];
      const Where w = locate(p, unit);
      const bool reduce = p.splitK > 1 || p.accumulate;
      if (live) live = __all_sync(0xffffffffu, mbarWait(&accFull[buf], accPhase, err));
      if (live) {
        fenceAfter();
        const int row0 = w.mb * 2 * BM + (int)cr * BM + q * 32, colBase = w.nb * BN + half * 128;
        const bool addBias = MODE != MODE_DUAL && args.bias != nullptr && w.first;
        if (addBias) {  // this warp's 128 bias values, once per tile, as fp32 in shared memory (columns past N read as 0)
          const __nv_bfloat16 *bias = (const __nv_bfloat16 *)args.bias;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int cidx = colBase + j * 32 + lane;
            biasW[j * 32 + lane] = cidx < p.N ? __bfloat162float(bias[cidx]) : 0.f;
          }
          __syncwarp();
        }
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += 32) {
          if (colBase + c0 >= p.N || row0 >= p.M) break;
          uint32_t r[32];
          tmemLd32(tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + half * 128 + c0), r);
          if (MODE == MODE_GELU) {
            // both staging blocks of this warp are used per step: the product goes into the first, the activation
            // into the second, and one thread hands both to the TMA unit
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            tmemLdWait();
            uint4 *stgPre = (uint4 *)stgBase, *stgAct = (uint4 *)(stgBase + STG_BYTES);
#pragma unroll
            for (int v = 0; v < 4; v++) {
              uint4 o;
              o.x = pack2(__uint_as_float(r[8 * v + 0]), __uint_as_float(r[8 * v + 1]));
              o.y = pack2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
              o.z = pack2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
              o.w = pack2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
              stgPre[lane * 4 + (v ^ ((lane >> 1) & 3))] = o;
            }
            const float4 *bv = (const float4 *)(biasW + c0);
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const float4 f = addBias ? bv[j] : make_float4(0.f, 0.f, 0.f, 0.f);
              r[4 * j + 0] = __float_as_uint(geluTanh(__uint_as_float(r[4 * j + 0]) + f.x));
              r[4 * j + 1] = __float_as_uint(geluTanh(__uint_as_float(r[4 * j + 1]) + f.y));
              r[4 * j + 2] = __float_as_uint(geluTanh(__uint_as_float(r[4 * j + 2]) + f.z));
              r[4 * j + 3] = __float_as_uint(geluTanh(__uint_as_float(r[4 * j + 3]) + f.w));
            }
#pragma unroll
            for (int v = 0; v < 4; v++) {
              uint4 o;
              o.x = pack2(__uint_as_float(r[8 * v + 0]), __uint_as_float(r[8 * v + 1]));
              o.y = pack2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
              o.z = pack2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
              o.w = pack2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
              stgAct[lane * 4 + (v ^ ((lane >> 1) & 3))] = o;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                           ::"l"(&p.c), "r"(colBase + c0), "r"(row0), "r"(smemAddr(stgPre)) : "memory");
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                           ::"l"(&args.c2), "r"(colBase + c0), "r"(row0), "r"(smemAddr(stgAct)) : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            chunkNo++;
            continue;
          }
          // the staging block about to be refilled must have been read out by the TMA unit
          if (lane == 0) {
            if (STG_DEPTH == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          }
          __syncwarp();
          tmemLdWait();
          if (addBias) {
            const float4 *bv = (const float4 *)(biasW + c0);  // same address in every lane: broadcast reads
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const float4 f = bv[j];
              r[4 * j + 0] = __float_as_uint(__uint_as_float(r[4 * j + 0]) + f.x);
              r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + f.y);
              r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + f.z);
              r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + f.w);
            }
          }
          uint4 *stg = (uint4 *)(stgBase + (chunkNo % STG_DEPTH) * STG_BYTES);
#pragma unroll
          for (int v = 0; v < 4; v++) {
            uint4 o;
            o.x = pack2(__uint_as_float(r[8 * v + 0]), __uint_as_float(r[8 * v + 1]));
            o.y = pack2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
            o.z = pack2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
            o.w = pack2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
            stg[lane * 4 + (v ^ ((lane >> 1) & 3))] = o;  // row = lane (64 bytes), 16-byte chunk XOR bits 1-2 of the row
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> the TMA unit's reads
          __syncwarp();
          if (lane == 0) {
            if (reduce)
              asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];"
                           ::"l"(&p.c), "r"(colBase + c0), "r"(row0), "r"(smemAddr(stg)) : "memory");
            else
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                           ::"l"(&p.c), "r"(colBase + c0), "r"(row0), "r"(smemAddr(stg)) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
          chunkNo++;
        }
        fenceBefore();
        __syncwarp();
        if (lane == 0) mbarArriveRemote(mapToCta(smemAddr(&accEmpty[buf]), 0));
      }
      if (++buf == 2) { buf = 0; accPhase ^= 1; }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every block has reached C
  }

  // ---- tear-down: nobody leaves, and no TMEM is freed, while the peer may still read this CTA's shared memory,
  // write its TMEM or arrive on its barriers
  fenceBefore();
  __syncthreads();
  clusterSync();
  fenceAfter();
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(512) : "memory");
}

}  // namespace

// 0 = never, 1 = when the shape suits (default), 2 = whenever the kernel can take the shape.
extern "C" int fcxGemmPairMode() {
  static const int mode = [] {
    const char *e = getenv("FLAGCX_GEMM_2SM");
    return e ? std::max(0, std::min(2, atoi(e))) : 1;
  }();
  return mode;
}

// Whether the pair kernel is the better choice for this shape: by the waves of tiles that either kernel needs, times what
// a K block of its tile costs; the pair kernel has to win clearly, since half-empty pair tiles waste both SMs.
// `cut`: the pieces of K that the launch asks for (0: the launcher's own choice, 1: K stays whole).
// `bn`: the tile width of the one-CTA kernel, for when it is that.
extern "C" int fcxGemmChoose(int M, int N, int K, int sms, int cut, int *bn) {
  const double tile = fcxGemmTileCostCut(M, N, K, sms, cut, bn);
  const int mode = fcxGemmPairMode();
  if (mode == 0 || M < 129 || K < 8) return 0;
  return mode == 2 || fcxGemmPairCostCut(M, N, K, sms / 2, cut) <= 0.85 * tile;
}
extern "C" int fcxGemmPairSuitsCut(int M, int N, int K, int cut) { return fcxGemmChoose(M, N, K, fcxhost::smCount(), cut, nullptr); }
extern "C" int fcxGemmPairSuits(int M, int N, int K) { return fcxGemmPairSuitsCut(M, N, K, 0); }

static bool fillProb(PairProb *p, const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int ldc, int aMN, int bMN, int group,
                     char *detail, size_t detailLen) {
  const bool okA = aMN ? makeTileMap(&p->a, a, K, M, lda, BK, 2) : makeTileMap(&p->a, a, M, K, lda, BM, 2);
  const bool okB = bMN ? makeTileMap(&p->b, b, K, N, ldb, BK, 2) : makeTileMap(&p->b, b, N, K, ldb, BNH, 2);
  const bool okC = makeStoreMap(&p->c, c, M, N, ldc);
  if (!okA || !okB || !okC) {
    if (detail)
      snprintf(detail, detailLen, "tensor map of %s refused (pair kernel, M %d N %d K %d)", !okA ? "operand A" : !okB ? "operand B" : "C", M, N, K);
    return false;
  }
  p->M = M; p->N = N; p->K = K; p->aMN = aMN; p->bMN = bMN; p->group = group;
  p->units = ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN);
  p->splitK = 1;
  return true;
}

template <int MODE>
static cudaError_t launchPair(const PairArgs &args, int pairs, cudaStream_t s) {
  static fcxhost::OncePerDevice once;
  const cudaError_t e = once([] { return cudaFuncSetAttribute(fcxGemmPairKernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES); });
  if (e != cudaSuccess) return e;
  return fcxpdl::launchPdl(fcxGemmPairKernel<MODE>, 2 * pairs, THREADS, SMEM_BYTES, s, args);
}

extern "C" cudaError_t fcxGemmPairBf16(const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int ldc, int aMN, int bMN,
                                       const void *bias, int splitK, int accumulate, void *geluOut, int group, int *errFlag, cudaStream_t s,
                                       char *detail, size_t detailLen) {
  PairArgs args{};
  if (geluOut && (accumulate || ((uintptr_t)geluOut & 15))) return cudaErrorInvalidValue;
  const bool ok = fillProb(&args.prob[0], a, b, c, M, N, K, lda, ldb, ldc, aMN, bMN, group, detail, detailLen);
  if (!ok) return cudaErrorNotSupported;
  if (geluOut) {
    if (!makeStoreMap(&args.c2, geluOut, M, N, ldc)) return cudaErrorNotSupported;
    splitK = 1;  // the activation needs the whole sum
  }
  PairProb &p = args.prob[0];
  const int sms = fcxhost::smCount(), pairs = sms / 2;
  p.splitK = fcxGemmPieces(splitK, M, N, K, p.units, pairs, sms);
  p.units *= p.splitK;
  p.accumulate = accumulate;
  args.bias = bias;
  args.errFlag = errFlag;
  if (p.splitK > 1 && !accumulate) {
    cudaError_t e = cudaMemsetAsync(c, 0, ((size_t)(M - 1) * ldc + N) * 2, s);
    if (e != cudaSuccess) return e;
  }
  const cudaError_t e = geluOut ? launchPair<MODE_GELU>(args, std::min(p.units, pairs), s) : launchPair<MODE_PLAIN>(args, std::min(p.units, pairs), s);
  if (e != cudaSuccess && detail)
    snprintf(detail, detailLen, "pair kernel launch: %s (M %d N %d K %d splitK %d units %d)", cudaGetErrorString(e), M, N, K, p.splitK, p.units);
  return e;
}

// How two products of units0 / units1 tiles with nK0 / nK1 K blocks each share one launch of `workers` workers: the K pieces
// of both (never more than either is cut into in a launch of its own), which one goes first (the one with the longer units;
// swap = the second product) and how many short units make up for a long one.  Every choice is tried; the time of a choice is
// that of its busiest worker, in K blocks.  Returns 0 when two launches would be done sooner.
extern "C" int fcxGemmDualPlan(int units0, int nK0, int alone0, int units1, int nK1, int alone1, int workers, int *split0, int *split1, int *swap,
                               int *extra) {
  auto pieces = [](int nK, int s) { const int per = (nK + s - 1) / s; return (nK + per - 1) / per; };
  double best = 0;
  int bestTime = 0;
  for (int a = 1; a <= alone0; a++)
    for (int b = 1; b <= alone1; b++) {
      if (pieces(nK0, a) != a || pieces(nK1, b) != b) continue;
      int len[2] = {(nK0 + a - 1) / a, (nK1 + b - 1) / b}, n[2] = {units0 * a, units1 * b};
      const int sw = len[1] > len[0], P = std::min(workers, n[0] + n[1]);
      if (sw) { std::swap(len[0], len[1]); std::swap(n[0], n[1]); }
      const int rem = n[0] % P;
      for (int ex = rem ? len[0] / len[1] : 0; ex <= (rem ? len[0] / len[1] + 1 : 0); ex++) {
        const int uniform = std::max(0, n[1] - ex * (P - rem));  // short units that go round all workers
        // the busiest workers are the first of those with one long unit more and the first of the others
        auto shorts = [&](int me) { return uniform > me ? (uniform - me + P - 1) / P : 0; };
        int time = (n[0] / P) * len[0] + (std::min(ex, (n[1] + P - rem - 1) / (P - rem)) + shorts(rem)) * len[1];
        if (rem) time = std::max(time, (n[0] / P + 1) * len[0] + shorts(0) * len[1]);
        const double cost = time * (1.0 + 0.02 * (a - 1 + b - 1));  // pieces are added in memory
        if (best == 0 || cost < best) {
          best = cost;
          bestTime = time;
          *split0 = a; *split1 = b; *swap = sw; *extra = ex;
        }
      }
    }
  const int apart = (units0 * alone0 + workers - 1) / workers * ((nK0 + alone0 - 1) / alone0) +
                    (units1 * alone1 + workers - 1) / workers * ((nK1 + alone1 - 1) / alone1);
  return bestTime <= apart;
}

// Whether `workers` workers visit every unit of a launch exactly once; the longest worker's time in `longest` (a unit of the
// first product takes len0, of the second len1).
extern "C" int fcxGemmUnitsCovered(int workers, int n0, int n1, int extra, int len0, int len1, int *longest) {
  std::vector<int> seen0(n0, 0), seen1(n1, 0);
  *longest = 0;
  for (int w = 0; w < workers; w++) {
    UnitIter it(w, workers, n0, n1, extra);
    int prob, unit, time = 0;
    while (it.next(&prob, &unit)) {
      if (unit < 0 || unit >= (prob ? n1 : n0)) return 0;
      (prob ? seen1 : seen0)[unit]++;
      time += prob ? len1 : len0;
    }
    *longest = std::max(*longest, time);
  }
  for (int c : seen0)
    if (c != 1) return 0;
  for (int c : seen1)
    if (c != 1) return 0;
  return 1;
}

// dx[T,I] = dy[T,O] w[O,I] and dw[O,I] (+)= dy^T x in one launch, for products that both suit the pair kernel.  Returns
// cudaErrorNotSupported when two launches would be done sooner.
extern "C" cudaError_t fcxGemmBackwardPair(const void *dy, const void *w, const void *x, void *dx, void *dw, int T, int I, int O, int lddy, int ldw,
                                           int ldx, int accumulate, int groupX, int groupW, int *errFlag, cudaStream_t s) {
  PairArgs args{};
  PairProb px{}, pw{};
  if (!fillProb(&px, dy, w, dx, T, I, O, lddy, ldw, I, 0, 1, groupX, nullptr, 0) ||
      !fillProb(&pw, dy, x, dw, O, I, T, lddy, ldx, I, 1, 1, groupW, nullptr, 0))
    return cudaErrorNotSupported;
  const int nKx = (O + BK - 1) / BK, nKw = (T + BK - 1) / BK, sms = fcxhost::smCount(), pairs = sms / 2;
  int swap = 0;
  if (!fcxGemmDualPlan(pw.units, nKw, fcxGemmPieces(0, O, I, T, pw.units, pairs, sms), px.units, nKx,
                       fcxGemmPieces(0, T, I, O, px.units, pairs, sms), pairs, &pw.splitK, &px.splitK, &swap, &args.extra))
    return cudaErrorNotSupported;
  pw.accumulate = accumulate;
  for (PairProb *p : {&px, &pw}) {
    p->units *= p->splitK;
    if (p->splitK > 1 && !p->accumulate) {
      cudaError_t e = cudaMemsetAsync(p == &px ? dx : dw, 0, (size_t)p->M * p->N * 2, s);
      if (e != cudaSuccess) return e;
    }
  }
  args.prob[0] = swap ? px : pw;
  args.prob[1] = swap ? pw : px;
  args.errFlag = errFlag;
  return launchPair<MODE_DUAL>(args, std::min(px.units + pw.units, pairs), s);
}

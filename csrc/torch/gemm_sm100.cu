// bf16 GEMM family on the 5th-generation tensor cores (tcgen05 + TMEM + TMA),
// written for sm_100a, with communication fused into the same kernel:
//
//   mode PLAIN   C[M,N] = A[M,K] * B[N,K]^T
//   mode AG      all-gather -> GEMM: A is the concatenation of every rank's
//                [M/n, K] block.  Dedicated "comm" CTAs push this rank's block
//                into every peer's gathered buffer over NVLink (plain stores)
//                and raise one flag per 128-row block; the GEMM CTAs start
//                with the local block, read in place through its own tensor
//                map, and consume remote blocks as their flags arrive, so
//                the transfer hides behind the math.
//   mode RS      GEMM -> reduce-scatter: every finished 128x256 tile is
//                written straight from TMEM (through registers) into the
//                staging area of the rank that owns those rows, tiles owned by
//                other ranks first, then an arrival counter is raised; after
//                its last tile each CTA turns to the reduction of the tiles
//                this rank owns (sum of the n partial tiles, fp32) as their
//                counters fill.
//
// The reference has no GEMM and no fused path: its users run a vendor
// all-gather / reduce-scatter and a vendor GEMM back to back.
//
// Structure (one CTA per SM, 256 threads, persistent over tiles):
//   warp 0    TMA producer: cp.async.bulk.tensor loads of A (128x64) and B
//             (256x64) tiles, 128-byte swizzle, 4-stage mbarrier pipeline.
//             All loads read this GPU's own memory and none is multicast.
//   warp 1    MMA issuer: one elected lane issues tcgen05.mma (M128 N256 K16,
//             bf16 x bf16 -> fp32) into one of two TMEM accumulators,
//             tcgen05.commit releases smem stages / publishes the accumulator.
//   warp 2    allocates and frees the 512 TMEM columns.
//   warps 4-7 epilogue: tcgen05.ld (32 lanes x 32 columns per warp and step),
//             fp32 -> bf16, transposed through shared memory so that global
//             stores (possibly into a peer) cover whole 128-byte lines.
// Every wait (mbarrier, flag, counter) is bounded: after the limit the kernel
// records an error, drains, frees its TMEM and returns.
#include "../kernels/prims.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_state.h"
#include "gemm_sm100.h"
#include "gemm_units.h"
#include "pdl.cuh"
#include "tcgen05.cuh"

namespace {

using namespace fcxmma;

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int EPI_BYTES = 4 * 32 * 128;  // per epilogue warp: 32 rows x 64 bf16
constexpr int BIAS_BYTES = 4 * 256 * 4;  // per epilogue warp: the tile's bias values as fp32
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + BIAS_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
constexpr int THREADS = 256;

// Instruction descriptor: D fp32, A/B bf16, both K-major, M = 128, N = 256.
__device__ __forceinline__ uint32_t instrDesc(int bn, int aMN = 0, int bMN = 0) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(aMN ? 1 : 0) << 15) | ((uint32_t)(bMN ? 1 : 0) << 16) |
         ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
constexpr int MN_BLOCK_BYTES = 64 * BK * 2;  // one 64-column block of an MN-major tile: BK lines of 128 bytes

// Tile t of this CTA's sequence -> (row block, column block).  Row blocks are
// visited in rotated order so that (AG) the local block comes first and (RS)
// the blocks this rank owns come last.
__device__ __forceinline__ void tileCoord(const FcxGemmParams &p, int nM, int t, int *mb, int *nb) {
  const int nN = (p.N + p.bn - 1) / p.bn;
  int g;
  if (p.group > 0) {
    // Row blocks in bands of `group`; inside a band the row block changes fastest, so the CTAs of one wave
    // share a few A row blocks and a few B column blocks and both stay in L2.
    const int perBand = p.group * nN, band = t / perBand, first = band * p.group;
    const int rowsHere = min(p.group, nM - first), within = t - band * perBand;
    g = first + within % rowsHere;
    *nb = within / rowsHere;
  } else {
    g = t / nN;
    *nb = t % nN;
  }
  *mb = (g + p.rotate) % nM;  // AG: the local rows first; RS: the rows this rank owns last
}

// The second of two independent products in one launch (DUAL: the input and weight gradients of a linear layer).
struct SecondProduct {
  CUtensorMap a, b;
  FcxGemmParams p;
  int extra;
};

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1) fcxGemmKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                                                            const __grid_constant__ CUtensorMap tmALocal, const __grid_constant__ FcxGemmParams p0,
                                                            const FcxDevComm dc, const __grid_constant__ SecondProduct second) {
  constexpr bool PLAIN = MODE == FCX_GEMM_PLAIN || MODE == FCX_GEMM_DUAL;
  extern __shared__ uint8_t smemRaw[];
  const int warp = warpIndex(), lane = threadIdx.x & 31;
  volatile int *err = p0.errFlag;

  // ------------------------------------------------------------ communication CTAs (AG mode only)
  if (MODE == FCX_GEMM_AG && (int)blockIdx.x >= p0.gemmCtas) {
    // This rank's [rowsPerRank, K] block goes, 128 rows at a time, to every rank's gathered buffer
    // (this rank's own copy included); one flag per destination and 128-row block.
    const int commCta = blockIdx.x - p0.gemmCtas, nComm = gridDim.x - p0.gemmCtas;
    const int n = dc.nranks, me = dc.rank;
    const int blocksPerRank = p0.rowsPerRank / BM;
    const size_t blockBytes = (size_t)BM * p0.K * 2;
    const int work = blocksPerRank * (n - 1);  // (remote destination, block) pairs; the local block is read where it lies
    for (int w = commCta; w < work; w += nComm) {
      // destinations rotate so that the ranks do not all write to the same GPU at once:
      // step k goes to rank me-k, so every rank receives from rank+1, rank+2, ... which is the
      // order in which its GEMM CTAs consume the remote blocks
      const int k = 1 + w / blocksPerRank, b = w % blocksPerRank;
      const int dst = (me - k + n) % n;
      const char *src = (const char *)p0.aLocal + (size_t)b * blockBytes;
      char *d = dc.heap[dst] + p0.gatherOff + ((size_t)me * blocksPerRank + b) * blockBytes;
      const uint4 *s4 = (const uint4 *)src;
      uint4 *d4 = (uint4 *)d;
      const size_t nvec = blockBytes / 16;
      size_t i = threadIdx.x;
      for (; i + 3 * THREADS < nvec; i += 4 * THREADS) {
        uint4 a = s4[i], bb = s4[i + THREADS], c = s4[i + 2 * THREADS], e = s4[i + 3 * THREADS];
        d4[i] = a; d4[i + THREADS] = bb; d4[i + 2 * THREADS] = c; d4[i + 3 * THREADS] = e;
      }
      for (; i < nvec; i += THREADS) d4[i] = s4[i];
      __syncthreads();
      if (threadIdx.x == 0) {
        uint64_t *flag = (uint64_t *)(dc.heap[dst] + p0.flagOff) + (size_t)me * blocksPerRank + b;
        fcxdev::stRelease(flag, p0.epoch);
      }
    }
    return;
  }

  // ------------------------------------------------------------ GEMM CTAs
  uint8_t *tiles = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t *epiStage = tiles + STAGES * STAGE_BYTES;
  float *biasStage = (float *)(epiStage + EPI_BYTES);
  uint64_t *bars = (uint64_t *)(epiStage + EPI_BYTES + BIAS_BYTES);
  uint64_t *fullBar = bars, *emptyBar = bars + STAGES, *tmemFull = bars + 2 * STAGES, *tmemEmpty = bars + 2 * STAGES + 2;
  uint32_t *tmemBaseSlot = (uint32_t *)(bars + 2 * STAGES + 4);

  if (MODE == FCX_GEMM_PLAIN && p0.mPtr) fcxpdl::pdlWait();  // the row count comes from the kernel before
  const int rows0 = p0.mPtr ? min(*p0.mPtr, p0.M) : p0.M;  // the row count may live on the device
  const int gemmCtas = (MODE == FCX_GEMM_AG) ? p0.gemmCtas : gridDim.x;
  // Unit of a product (tile, and piece of K when it is cut) -> where it lies.
  struct Where {
    int mb, nb, kLo, kHi;
    bool first;
  };
  auto splitOf = [](const FcxGemmParams &p) { return PLAIN && p.splitK > 1 ? p.splitK : 1; };
  auto locate = [&](const FcxGemmParams &p, int rows, int u) {
    Where w;
    const int nM = (rows + BM - 1) / BM, nK = (p.K + BK - 1) / BK, sk = splitOf(p), kPer = (nK + sk - 1) / sk, piece = u % sk;
    tileCoord(p, nM, u / sk, &w.mb, &w.nb);
    w.kLo = piece * kPer;
    w.kHi = min(nK, w.kLo + kPer);
    w.first = piece == 0;
    return w;
  };
  auto unitsOf = [&](const FcxGemmParams &p, int rows) { return ((rows + BM - 1) / BM) * ((p.N + p.bn - 1) / p.bn) * splitOf(p); };
  UnitIter it(blockIdx.x, gemmCtas, unitsOf(p0, rows0), MODE == FCX_GEMM_DUAL ? unitsOf(second.p, second.p.M) : 0,
              MODE == FCX_GEMM_DUAL ? second.extra : 0);
  int which = 0, unit = 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbarInit(&fullBar[s], 1); mbarInit(&emptyBar[s], 1); }
    for (int b = 0; b < 2; b++) { mbarInit(&tmemFull[b], 1); mbarInit(&tmemEmpty[b], 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemBaseSlot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fenceBefore();
  __syncthreads();
  fenceAfter();
  const uint32_t tmemBase = *tmemBaseSlot;
  if (PLAIN) {
    fcxpdl::pdlRelease();
    fcxpdl::pdlWait();  // everything above touches only this CTA's own memories
  }

  if (warp == 0) {
    // ---- TMA producer
    if (electOne()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      while (ok && it.next(&which, &unit)) {
        const FcxGemmParams &p = MODE == FCX_GEMM_DUAL && which ? second.p : p0;
        const Where w = locate(p, MODE == FCX_GEMM_DUAL ? p.M : rows0, unit);
        const int bn = p.bn;
        const int mb = w.mb, nb = w.nb;
        const CUtensorMap *mapA = MODE == FCX_GEMM_DUAL && which ? &second.a : &tmA, *mapB = MODE == FCX_GEMM_DUAL && which ? &second.b : &tmB;
        int rowA = mb * BM;
        if (MODE == FCX_GEMM_AG) {
          const int blocksPerRank = p.rowsPerRank / BM, owner = mb / blocksPerRank;
          if (owner == dc.rank) {
            // this rank's own rows are read straight from the caller's tensor
            mapA = &tmALocal;
            rowA = (mb - owner * blocksPerRank) * BM;
          } else {
            // rows of block mb must have arrived in the gathered buffer
            const uint64_t *flag = (const uint64_t *)(dc.heap[dc.rank] + p.flagOff) + mb;
            ok = fcxdev::waitGe(dc, flag, p.epoch, owner, FCX_WAIT_DEVAPI, blockIdx.x, p.epoch);
            if (!ok) { *err = 1; break; }
            asm volatile("fence.proxy.async;" ::: "memory");  // remote generic-proxy writes -> this CTA's TMA reads
          }
        }
        for (int kb = w.kLo; kb < w.kHi; kb++) {
          if (!mbarWait(&emptyBar[stage], phase ^ 1, err)) { ok = false; break; }
          mbarExpectTx(&fullBar[stage], A_BYTES + bn * BK * 2);
          uint8_t *sa = tiles + stage * STAGE_BYTES, *sb = sa + A_BYTES;
          if (PLAIN && p.aMN) {
            // stored [K, M]: two blocks of 64 columns (M) x BK lines (K)
            for (int j = 0; j < BM / 64; j++) tmaLoad2d(sa + j * MN_BLOCK_BYTES, mapA, rowA + j * 64, kb * BK, &fullBar[stage]);
          } else {
            tmaLoad2d(sa, mapA, kb * BK, rowA, &fullBar[stage]);
          }
          if (PLAIN && p.bMN) {
            for (int j = 0; j < bn / 64; j++) tmaLoad2d(sb + j * MN_BLOCK_BYTES, mapB, nb * bn + j * 64, kb * BK, &fullBar[stage]);
          } else {
            tmaLoad2d(sb, mapB, kb * BK, nb * bn, &fullBar[stage]);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the warp waits as one, one lane issues
    int stage = 0, buf = 0;
    uint32_t phase = 0, accPhase = 0;
    bool ok = true;
    while (ok && it.next(&which, &unit)) {
      const FcxGemmParams &p = MODE == FCX_GEMM_DUAL && which ? second.p : p0;
      const Where w = locate(p, MODE == FCX_GEMM_DUAL ? p.M : rows0, unit);
      const int bn = p.bn;
      const bool aMN = PLAIN && p.aMN, bMN = PLAIN && p.bMN;
      const uint32_t idesc = instrDesc(bn, aMN, bMN);
      if (!__all_sync(0xffffffffu, mbarWait(&tmemEmpty[buf], accPhase ^ 1, err))) break;
      fenceAfter();
      const uint32_t dTmem = tmemBase + (uint32_t)buf * 256;
      for (int kb = w.kLo; kb < w.kHi; kb++) {
        if (!__all_sync(0xffffffffu, mbarWait(&fullBar[stage], phase, err))) { ok = false; break; }
        fenceAfter();
        if (electOne()) {
          const uint32_t sa = smemAddr(tiles + stage * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; k++) {
            // K-major: 16 bf16 = 32 bytes further along K inside the 128-byte swizzle row;
            // MN-major: 16 K indices = two eight-line groups = 2048 bytes further
            const uint64_t da = aMN ? smemDescMN(sa + k * 2048, MN_BLOCK_BYTES) : smemDesc(sa + k * 32);
            const uint64_t db = bMN ? smemDescMN(sb + k * 2048, MN_BLOCK_BYTES) : smemDesc(sb + k * 32);
            mmaF16(dTmem, da, db, idesc, (kb > w.kLo || k > 0) ? 1u : 0u);
          }
          mmaCommit(&emptyBar[stage]);                         // the stage may be refilled once these MMAs have read it
          if (kb + 1 == w.kHi) mmaCommit(&tmemFull[buf]);      // accumulator complete
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (++buf == 2) { buf = 0; accPhase ^= 1; }
    }
  } else if (warp >= 4) {
    // ---- epilogue: warp w owns TMEM lanes [32*(w%4), +32) = rows of the tile.
    // A wait that gives up turns the warp "dead": it keeps walking the tile list (so that the
    // barriers it shares with the other epilogue warps stay matched) but touches nothing.
    const int q = warp & 3;
    int buf = 0;
    uint32_t accPhase = 0;
    bool live = true;
    while (it.next(&which, &unit)) {
      const FcxGemmParams &p = MODE == FCX_GEMM_DUAL && which ? second.p : p0;
      const Where w = locate(p, MODE == FCX_GEMM_DUAL ? p.M : rows0, unit);
      const int bn = p.bn;
      const int mb = w.mb, nb = w.nb, Mrows = MODE == FCX_GEMM_DUAL ? p.M : rows0, nN = (p.N + bn - 1) / bn;
      if (live) live = __all_sync(0xffffffffu, mbarWait(&tmemFull[buf], accPhase, err));
      if (live) {
        fenceAfter();
        // first row of this warp's 32-row band and where it goes
        const int row0 = mb * BM + q * 32;
        __nv_bfloat16 *dst0;
        size_t ldd;
        if (MODE == FCX_GEMM_RS) {
          const int owner = min(row0 / p.rowsPerRank, dc.nranks - 1), lrow0 = row0 - owner * p.rowsPerRank;
          dst0 = (__nv_bfloat16 *)(dc.heap[owner] + p.stageOff) + ((size_t)dc.rank * p.rowsPerRank + lrow0) * p.N;
          ldd = p.N;
        } else {
          dst0 = (__nv_bfloat16 *)p.c + (size_t)row0 * p.ldc;
          ldd = p.ldc;
        }
        // The accumulator comes out of TMEM one row per lane; a transposition through
        // shared memory (32 rows x 128 bytes per warp, 16-byte chunks XOR-swizzled by row)
        // turns that into stores where 8 lanes write one full 128-byte line of a row.
        uint4 *stg = (uint4 *)(epiStage + (size_t)q * 32 * 128);
        // the tile's bias values, once per tile and warp, as fp32 in shared memory (columns past N read as 0)
        const bool addBias = PLAIN && p.bias != nullptr && w.first;
        float *biasW = biasStage + q * 256;
        if (addBias) {
          const __nv_bfloat16 *bias = (const __nv_bfloat16 *)p.bias;
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int cidx = nb * bn + j * 32 + lane;
            biasW[j * 32 + lane] = (j * 32 < bn && cidx < p.N) ? __bfloat162float(bias[cidx]) : 0.f;
          }
          __syncwarp();
        }
#pragma unroll 1
        for (int c0 = 0; c0 < bn; c0 += 64) {
          uint32_t r[32];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            tmemLd32(tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 256 + c0 + 32 * h), r);
            tmemLdWait();
            if (addBias) {
              // every lane holds one row and the same 32 columns: broadcast reads of the staged bias values
              const float4 *bv = (const float4 *)(biasW + c0 + 32 * h);
#pragma unroll
              for (int j = 0; j < 8; j++) {
                const float4 f = bv[j];
                r[4 * j + 0] = __float_as_uint(__uint_as_float(r[4 * j + 0]) + f.x);
                r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + f.y);
                r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + f.z);
                r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + f.w);
              }
            }
#pragma unroll
            for (int v = 0; v < 4; v++) {
              uint4 o;
              o.x = pack2(__uint_as_float(r[8 * v + 0]), __uint_as_float(r[8 * v + 1]));
              o.y = pack2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
              o.z = pack2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
              o.w = pack2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
              stg[lane * 8 + ((4 * h + v) ^ (lane & 7))] = o;
            }
          }
          __syncwarp();
          const int col = nb * bn + c0 + (lane & 7) * 8;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int rr = i * 4 + (lane >> 3);
            uint4 o = stg[rr * 8 + ((lane & 7) ^ (rr & 7))];
            if (row0 + rr < Mrows) {
              __nv_bfloat16 *d = dst0 + (size_t)rr * ldd + col;
              if (PLAIN && (p.splitK > 1 || p.accumulate)) {
                // one K piece of several, or a contribution to a gradient that is being accumulated: added into C
                const uint32_t *w = (const uint32_t *)&o;
                for (int j = 0; j < 4; j++)
                  if (col + 2 * j + 1 < p.N || (col + 2 * j < p.N && (p.N & 1) == 0))
                    asm volatile("red.global.add.noftz.bf16x2 [%0], %1;" ::"l"(d + 2 * j), "r"(w[j]) : "memory");
              } else if (col + 8 <= p.N) *(uint4 *)d = o;
              else {
                const __nv_bfloat16 *e = (const __nv_bfloat16 *)&o;
                for (int j = 0; j < 8 && col + j < p.N; j++) d[j] = e[j];
              }
            }
          }
          __syncwarp();
        }
        fenceBefore();
        __syncwarp();
        if (lane == 0) mbarArrive(&tmemEmpty[buf]);
      }
      if (MODE == FCX_GEMM_RS) {
        // publish the tile to its owner: every epilogue warp fences its stores, then one thread counts the tile
        __threadfence_system();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (live && warp == 4 && lane == 0) {
          const int owner = (mb * BM) / p.rowsPerRank, lmb = (mb * BM % p.rowsPerRank) / BM;
          uint64_t *cnt = (uint64_t *)(dc.heap[owner] + p.flagOff) + (size_t)lmb * nN + nb;
          asm volatile("red.release.sys.global.add.u64 [%0], %1;" ::"l"(cnt), "l"((uint64_t)1) : "memory");
        }
      }
      if (++buf == 2) { buf = 0; accPhase ^= 1; }
    }
  }

  // ------------------------------------------------------------ tear-down
  fenceBefore();
  __syncthreads();
  fenceAfter();
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(512) : "memory");

  // ------------------------------------------------------------ RS: reduce the tiles this rank owns
  if (MODE == FCX_GEMM_RS) {
    const FcxGemmParams &p = p0;
    const int nN = (p.N + BN - 1) / BN;
    const int n = dc.nranks, lBlocks = p.rowsPerRank / BM;
    const int items = lBlocks * nN;
    const uint64_t want = p.epoch * (uint64_t)n;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
      const int lmb = it / nN, nb = it % nN;
      bool ok = true;
      if (threadIdx.x == 0) {
        const uint64_t *cnt = (const uint64_t *)(dc.heap[dc.rank] + p.flagOff) + (size_t)lmb * nN + nb;
        ok = fcxdev::waitGe(dc, cnt, want, -1, FCX_WAIT_DEVAPI, blockIdx.x, p.epoch);
        if (!ok) *err = 1;
      }
      if (!__syncthreads_and(ok)) break;
      // 128 x 256 outputs, 8 per thread step: thread handles 16-byte vectors
      const int colsHere = min(BN, p.N - nb * BN);
      const int vecPerRow = colsHere / 8;
      const __nv_bfloat16 *stage = (const __nv_bfloat16 *)(dc.heap[dc.rank] + p.stageOff);
      for (int v = threadIdx.x; v < BM * vecPerRow; v += THREADS) {
        const int r = v / vecPerRow, cv = v % vecPerRow;
        const int lrow = lmb * BM + r;
        if (lrow >= p.rowsPerRank) break;
        const size_t off = (size_t)lrow * p.N + nb * BN + cv * 8;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = 0; s < n; s++) {
          uint4 x = *(const uint4 *)(stage + (size_t)s * p.rowsPerRank * p.N + off);
          const __nv_bfloat162 *h = (const __nv_bfloat162 *)&x;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            float2 f = __bfloat1622float2(h[j]);
            acc[2 * j] += f.x;
            acc[2 * j + 1] += f.y;
          }
        }
        uint4 o;
        o.x = pack2(acc[0], acc[1]); o.y = pack2(acc[2], acc[3]); o.z = pack2(acc[4], acc[5]); o.w = pack2(acc[6], acc[7]);
        *(uint4 *)((__nv_bfloat16 *)p.c + (size_t)lrow * p.ldc + nb * BN + cv * 8) = o;
      }
    }
  }
}

// ------------------------------------------------------------------ host side

// Row-major [rows, cols] bf16 matrix with `ld` elements between rows; box = [boxRows, 64 columns], 128-byte swizzle.
bool makeMap(CUtensorMap *m, const void *base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t boxRows) {
  return makeTileMap(m, base, rows, cols, ld, boxRows, 2);
}

template <int MODE>
cudaError_t launch(const CUtensorMap &a, const CUtensorMap &b, const FcxGemmParams &p, const FcxDevComm &dc, int grid, cudaStream_t s,
                   const CUtensorMap *aLocal = nullptr, const SecondProduct *second = nullptr) {
  static fcxhost::OncePerDevice once;
  const cudaError_t e = once([] { return cudaFuncSetAttribute(fcxGemmKernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES); });
  if (e != cudaSuccess) return e;
  SecondProduct none{};
  const CUtensorMap &al = aLocal ? *aLocal : a;
  const SecondProduct &q = second ? *second : none;
  // the kernels that exchange with peers are launched plainly: their first accesses are flags and peers' memory
  if (MODE == FCX_GEMM_PLAIN || MODE == FCX_GEMM_DUAL) return fcxpdl::launchPdl(fcxGemmKernel<MODE>, grid, THREADS, SMEM_BYTES, s, a, b, al, p, dc, q);
  fcxGemmKernel<MODE><<<grid, THREADS, SMEM_BYTES, s>>>(a, b, al, p, dc, q);
  return cudaGetLastError();
}

// Row blocks per band of the tile order (FLAGCX_GEMM_TILE_GROUP; 0 = plain row-major order).
int tileGroup(int nN) {
  static const int g = [] {
    const char *e = getenv("FLAGCX_GEMM_TILE_GROUP");
    return e ? std::max(0, atoi(e)) : -1;
  }();
  return g >= 0 ? g : (nN >= 24 ? 16 : 8);  // wide outputs: taller bands keep more of B in L2 per wave
}

// FLAGCX_GEMM_BN (64, 128, 256): columns per tile of the one-CTA kernel, for experiments.
int forcedBn() {
  static const int forced = [] {
    const char *e = getenv("FLAGCX_GEMM_BN");
    const int v = e ? atoi(e) : 0;
    return v == 64 || v == 128 || v == 256 ? v : 0;
  }();
  return forced;
}

// Columns per tile of the one-CTA kernel.  `cut`: the pieces that the caller will ask fcxGemmPickSplitK for (1: K stays whole).
int pickBn(int M, int N, int K, int sms, int cut) {
  int bn = 256;
  if (!forcedBn()) fcxGemmTileCostCut(M, N, K, sms, cut, &bn);
  return forcedBn() ? forcedBn() : bn;
}

// The same choice together with that of the kernel: whether CTA pairs are the better one.
bool choose(int M, int N, int K, int sms, int cut, int *bn) {
  const bool pair = fcxGemmChoose(M, N, K, sms, cut, bn) != 0;
  if (forcedBn()) *bn = forcedBn();
  return pair;
}

using fcxhost::smCount;

}  // namespace

extern "C" cudaError_t fcxGemmBf16(const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int ldc, int *errFlag,
                                   cudaStream_t s) {
  if (K % 8 || lda % 8 || ldb % 8 || ldc % 8 || M <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
  if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) return cudaErrorInvalidValue;
  CUtensorMap ma, mb;
  const int bn = pickBn(M, N, K, smCount(), 1);
  if (!makeMap(&ma, a, M, K, lda, BM) || !makeMap(&mb, b, N, K, ldb, bn)) return cudaErrorNotSupported;
  FcxGemmParams p{};
  p.M = M; p.N = N; p.K = K; p.c = c; p.ldc = ldc; p.errFlag = errFlag; p.rotate = 0; p.bn = bn; p.group = tileGroup((N + bn - 1) / bn);
  FcxDevComm dc{};
  int tiles = ((M + BM - 1) / BM) * ((N + bn - 1) / bn);
  return launch<FCX_GEMM_PLAIN>(ma, mb, p, dc, std::min(tiles, smCount()), s);
}

// Pieces to cut K into.  requested > 0: that many (at most one per K block, and no piece may be empty).  Otherwise: few
// tiles and a long K (the weight-gradient GEMMs: K = tokens) are cut so that the pieces fill whole waves; a split into
// s pieces takes ceil(units * s / slots) waves of 1/s the length, and every extra piece costs some reduction traffic,
// counted as 3 % of a tile (1 % when K is very long).
extern "C" int fcxGemmPickSplitK(int requested, int units, int slots, int nK, int N) {
  int splitK = requested;
  if (splitK <= 0) {
    splitK = 1;
    const bool few = units < slots && nK >= 32;
    // more tiles than slots but a poor last wave and a very long K (the LM head's input gradient: 128 tiles on 74
    // pairs, K = 50304): zeroing C is noise against such a K, and the pieces stay long
    const bool longK = units >= slots && nK >= 256;
    if (few || longK) {
      const double base = (double)((units + slots - 1) / slots), piece = few ? 0.03 : 0.01;
      double best = 1.0;
      for (int sk = 2; sk <= 8 && nK / sk >= 8; sk++) {
        const double waves = (double)((units * sk + slots - 1) / slots);
        const double cost = waves / (sk * base) + piece * (sk - 1);
        if (cost < best - (splitK == 1 ? 0.05 : 0.0)) { best = cost; splitK = sk; }  // a first cut must pay clearly
      }
    }
  }
  if (N % 2) return 1;  // the partial results are added two columns at a time
  splitK = std::max(1, std::min(splitK, nK));
  const int kPer = (nK + splitK - 1) / splitK;
  return (nK + kPer - 1) / kPer;
}

// The pieces of K of one launch: those asked for, else the launcher's choice for `units` tiles on `slots` workers.  Each piece
// is rounded to bf16 once more where it is added in memory, so the choice of a kernel and tile must not cost exactness: K
// is never cut finer than by CTA pairs where the rows fill their 256-row blocks to 7 %, and by single CTAs with 256-column
// tiles elsewhere.  (The pair kernel counts half the slots and, with a half-empty last row block, less than half the tiles:
// 288 x 3392 x 3832 would be cut in 5 in place of 3.)
extern "C" int fcxGemmPieces(int requested, int M, int N, int K, int units, int slots, int sms) {
  const int nK = (K + BK - 1) / BK, pieces = fcxGemmPickSplitK(requested, units, slots, nK, N);
  if (requested > 0 || pieces == 1) return pieces;
  const int nN = (N + BN - 1) / BN, pairRows = (M + 2 * BM - 1) / (2 * BM);
  const bool fills = M > BM && N >= 192 && pairRows * 2 * BM <= 1.07 * M;
  const int most = fills ? fcxGemmPickSplitK(0, pairRows * nN, sms / 2, nK, N) : fcxGemmPickSplitK(0, (M + BM - 1) / BM * nN, sms, nK, N);
  return pieces <= most ? pieces : fcxGemmPickSplitK(most, units, slots, nK, N);
}

static double waveCost(int M, int N, int K, int units, int slots, int sms, int cut, double blockCost) {
  const int nK = (K + BK - 1) / BK, sk = fcxGemmPieces(cut, M, N, K, units, slots, sms);
  const int waves = (units * sk + slots - 1) / slots;
  return waves * ((nK + sk - 1) / sk) * blockCost * (1.0 + 0.03 * (sk - 1));
}

// Estimated clocks of the one-CTA kernel with its best tile width, and that width.  A 64-deep K block of a 128 x bn tile is
// bound by what one SM can fetch (16 KB of A and bn x 128 bytes of B at about 64 bytes a clock): 768, 512 and 384 clocks
// for 256, 128 and 64 columns.  Narrow tiles re-read A and never pay once 256-column tiles fill the SMs, but with few
// tiles they put more SMs to work on the same K steps.  `cut` is the launch's own: a sum that stays whole (1) keeps as many
// SMs busy as it has tiles, one that may be cut (0) fills them whatever its tiles are.  Uncut, measured: 512 x 1024 x 4096
// 20.2 / 21.9 / 24.9 us in 64 / 128 / 256 columns and 23.1 on CTA pairs; 640 x 3584 x 4096 38.2 / 24.4 / 28.6 and 25.3;
// 4096 x 1024 x 1792 33.2 / 20.6 / 15.0 and 13.9; 512 x 4096 x 1024 12.4 / 9.2 / 10.9 and 10.1.
extern "C" double fcxGemmTileCostCut(int M, int N, int K, int sms, int cut, int *bnOut) {
  const int nM = (M + BM - 1) / BM;
  const int widths[3] = {256, 128, 64};
  const double clocks[3] = {768, 512, 384};
  double best = 0;
  for (int i = 0; i < 3; i++) {
    const double c = waveCost(M, N, K, nM * ((N + widths[i] - 1) / widths[i]), sms, sms, cut, clocks[i]);
    if (i == 0 || c < 0.9 * best) {
      best = c;
      if (bnOut) *bnOut = widths[i];
    }
  }
  return best;
}

extern "C" double fcxGemmTileCost(int M, int N, int K, int sms, int *bnOut) { return fcxGemmTileCostCut(M, N, K, sms, 0, bnOut); }

// The same for the CTA-pair kernel: 32 KB per CTA and K block of a 256 x 256 tile.
extern "C" double fcxGemmPairCostCut(int M, int N, int K, int pairs, int cut) {
  return waveCost(M, N, K, ((M + 255) / 256) * ((N + 255) / 256), pairs, 2 * pairs, cut, 512);
}
extern "C" double fcxGemmPairCost(int M, int N, int K, int pairs) { return fcxGemmPairCostCut(M, N, K, pairs, 0); }

// What went wrong in the last fcxGemmBf16Ex call of this thread that did not return cudaSuccess.
static thread_local char gGemmDetail[256];
extern "C" const char *fcxGemmLastDetail() { return gGemmDetail; }

extern "C" cudaError_t fcxGemmBf16Opts(const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int ldc,
                                       const FcxGemmOpts *o, int *errFlag, cudaStream_t s) {
  const int aMN = o->aMN, bMN = o->bMN, accumulate = o->accumulate;
  const void *bias = o->bias;
  int splitK = o->splitK;
  if (K % 8 || lda % 8 || ldb % 8 || ldc % 8 || M <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
  if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) return cudaErrorInvalidValue;
  if ((aMN && M % 8) || (bMN && N % 8) || (bias && ((uintptr_t)bias & 1)) || (accumulate && N % 2)) return cudaErrorInvalidValue;
  gGemmDetail[0] = 0;
  cudaGetLastError();  // an error left behind by an earlier, unrelated call of this thread is not this launch's
  const int sms = smCount();
  int bn = 256;
  const bool pair = choose(M, N, K, sms, splitK, &bn);
  if (o->geluOut || (o->pair >= 0 ? o->pair > 0 : pair))  // CTA pairs on 256 x 256 tiles (gemm2_sm100.cu)
    return fcxGemmPairBf16(a, b, c, M, N, K, lda, ldb, ldc, aMN, bMN, bias, splitK, accumulate, o->geluOut, tileGroup((N + 255) / 256) / 2,
                           errFlag, s, gGemmDetail, sizeof gGemmDetail);
  CUtensorMap ma, mb;
  // K-major operand: rows = M (or N), box of 128 (bn) rows x 64 K; MN-major operand: rows = K, box of 64 lines x 64 columns
  const bool okA = aMN ? makeMap(&ma, a, K, M, lda, BK) : makeMap(&ma, a, M, K, lda, BM);
  const bool okB = bMN ? makeMap(&mb, b, K, N, ldb, BK) : makeMap(&mb, b, N, K, ldb, bn);
  if (!okA || !okB) {
    snprintf(gGemmDetail, sizeof gGemmDetail, "tensor map of operand %s refused (M %d N %d K %d lda %d ldb %d aMN %d bMN %d a %p b %p)",
             !okA ? "A" : "B", M, N, K, lda, ldb, aMN, bMN, a, b);
    return cudaErrorNotSupported;
  }
  FcxGemmParams p{};
  p.M = M; p.N = N; p.K = K; p.c = c; p.ldc = ldc; p.errFlag = errFlag; p.rotate = 0; p.bn = bn; p.group = tileGroup((N + bn - 1) / bn);
  p.aMN = aMN; p.bMN = bMN; p.bias = bias; p.accumulate = accumulate;
  const int tiles = ((M + BM - 1) / BM) * ((N + bn - 1) / bn);
  p.splitK = fcxGemmPieces(splitK, M, N, K, tiles, sms, sms);
  if (p.splitK > 1 && !accumulate) {
    cudaError_t e = cudaMemsetAsync(c, 0, ((size_t)(M - 1) * ldc + N) * 2, s);
    if (e != cudaSuccess) return e;
  }
  FcxDevComm dc{};
  cudaError_t e = launch<FCX_GEMM_PLAIN>(ma, mb, p, dc, std::min(tiles * p.splitK, sms), s);
  if (e != cudaSuccess)
    snprintf(gGemmDetail, sizeof gGemmDetail, "kernel launch: %s (M %d N %d K %d aMN %d bMN %d splitK %d grid %d)", cudaGetErrorString(e), M, N,
             K, aMN, bMN, p.splitK, std::min(tiles * p.splitK, sms));
  return e;
}

extern "C" cudaError_t fcxGemmBf16Ex(const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int ldc, int aMN, int bMN,
                                     const void *bias, int splitK, int *errFlag, cudaStream_t s) {
  FcxGemmOpts o{};
  o.aMN = aMN; o.bMN = bMN; o.bias = bias; o.splitK = splitK; o.accumulate = 0; o.pair = -1;
  return fcxGemmBf16Opts(a, b, c, M, N, K, lda, ldb, ldc, &o, errFlag, s);
}

extern "C" cudaError_t fcxGemmBf16DynM(const void *a, const void *b, void *c, int Mmax, const int *mPtr, int N, int K, int lda, int ldb, int ldc,
                                       int *errFlag, cudaStream_t s) {
  if (K % 8 || lda % 8 || ldb % 8 || ldc % 8 || Mmax <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
  CUtensorMap ma, mb;
  const int bn = pickBn(Mmax, N, K, smCount(), 1);
  if (!makeMap(&ma, a, Mmax, K, lda, BM) || !makeMap(&mb, b, N, K, ldb, bn)) return cudaErrorNotSupported;
  FcxGemmParams p{};
  p.M = Mmax; p.N = N; p.K = K; p.c = c; p.ldc = ldc; p.errFlag = errFlag; p.mPtr = mPtr; p.bn = bn; p.group = tileGroup((N + bn - 1) / bn);
  FcxDevComm dc{};
  int tiles = ((Mmax + BM - 1) / BM) * ((N + bn - 1) / bn);
  return launch<FCX_GEMM_PLAIN>(ma, mb, p, dc, std::min(tiles, smCount()), s);
}

// All-gather -> GEMM and GEMM -> reduce-scatter of one rank: there is nothing to exchange, so the plain GEMM writes the
// result itself (as CTA pairs where the shape suits) in place of a copy of the partial tiles in the staging area that is
// then read back.  K is not cut: the sums stay fp32 until the one rounding, as in the fused kernels.  `exchange` of the two
// entry points below takes the exchanging kernel all the same, with this GPU as its own peer: tests and profiles need it.
static cudaError_t oneRank(const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int ldc, int *errFlag, cudaStream_t s) {
  FcxGemmOpts o{};
  o.splitK = 1;
  o.pair = -1;
  return fcxGemmBf16Opts(a, b, c, M, N, K, lda, ldb, ldc, &o, errFlag, s);
}

extern "C" cudaError_t fcxAgGemmBf16(const FcxDevComm *dc, const void *aLocal, const void *gathered, size_t gatherOff, size_t flagOff,
                                     const void *b, void *c, int M, int N, int K, int ldb, int ldc, uint64_t epoch, int commCtas,
                                     int exchange, int *errFlag, cudaStream_t s) {
  const int n = dc->nranks;
  if (K % 8 || ldb % 8 || ldc % 8 || M % (n * BM) || commCtas < 1) return cudaErrorInvalidValue;
  if (n == 1 && !exchange) return oneRank(aLocal, b, c, M, N, K, K, ldb, ldc, errFlag, s);
  CUtensorMap ma, mb;
  const int bn = pickBn(M, N, K, std::max(1, smCount() - commCtas), 1);
  CUtensorMap mal;
  if (!makeMap(&ma, gathered, M, K, K, BM) || !makeMap(&mb, b, N, K, ldb, bn) || !makeMap(&mal, aLocal, M / n, K, K, BM))
    return cudaErrorNotSupported;
  FcxGemmParams p{};
  p.M = M; p.N = N; p.K = K; p.c = c; p.ldc = ldc; p.errFlag = errFlag; p.bn = bn; p.group = tileGroup((N + bn - 1) / bn);
  p.rowsPerRank = M / n;
  p.rotate = dc->rank * (p.rowsPerRank / BM);
  p.group = std::max(1, std::min(p.group, p.rowsPerRank / BM));  // a band never mixes rows of two ranks: they arrive at different times
  p.aLocal = aLocal; p.gatherOff = gatherOff; p.flagOff = flagOff; p.epoch = epoch;
  int tiles = (M / BM) * ((N + bn - 1) / bn);
  p.gemmCtas = std::max(1, std::min(tiles, smCount() - commCtas));
  return launch<FCX_GEMM_AG>(ma, mb, p, *dc, p.gemmCtas + commCtas, s, &mal);
}

extern "C" cudaError_t fcxGemmRsBf16(const FcxDevComm *dc, const void *a, const void *b, void *out, size_t stageOff, size_t flagOff, int M,
                                     int N, int K, int lda, int ldb, int ldc, uint64_t epoch, int exchange, int *errFlag, cudaStream_t s) {
  const int n = dc->nranks;
  if (K % 8 || lda % 8 || ldb % 8 || ldc % 8 || N % 8 || M % (n * BM)) return cudaErrorInvalidValue;
  if (n == 1 && !exchange) return oneRank(a, b, out, M, N, K, lda, ldb, ldc, errFlag, s);
  CUtensorMap ma, mb;
  if (!makeMap(&ma, a, M, K, lda, BM) || !makeMap(&mb, b, N, K, ldb, BN)) return cudaErrorNotSupported;
  FcxGemmParams p{};
  p.M = M; p.N = N; p.K = K; p.c = out; p.ldc = ldc; p.errFlag = errFlag; p.bn = BN;  // counters are laid out per 256 columns
  p.group = tileGroup((N + BN - 1) / BN);
  p.rowsPerRank = M / n;
  p.rotate = ((dc->rank + 1) % n) * (p.rowsPerRank / BM);
  p.stageOff = stageOff; p.flagOff = flagOff; p.epoch = epoch;
  int tiles = (M / BM) * ((N + BN - 1) / BN);
  return launch<FCX_GEMM_RS>(ma, mb, p, *dc, std::min(tiles, smCount()), s);
}

// The input and weight gradients of a linear layer in one launch: dx[T,I] = dy[T,O] w[O,I], dw[O,I] = dy^T x (added to dw
// with `accumulate`).  Returns cudaErrorNotSupported for sizes that are better off as two launches (one product on CTA
// pairs and the other not).
extern "C" cudaError_t fcxGemmBackwardBf16(const void *dy, const void *w, const void *x, void *dx, void *dw, int T, int I, int O, int lddy, int ldw,
                                           int ldx, int accumulate, int *errFlag, cudaStream_t s) {
  if (T % 8 || I % 8 || O % 8 || lddy % 8 || ldw % 8 || ldx % 8 || T <= 0 || I <= 0 || O <= 0) return cudaErrorNotSupported;
  if (((uintptr_t)dy | (uintptr_t)w | (uintptr_t)x | (uintptr_t)dx | (uintptr_t)dw) & 15) return cudaErrorNotSupported;
  cudaGetLastError();
  const int sms = smCount();
  int bnX = 256, bnW = 256;
  const bool pairX = choose(T, I, O, sms, 0, &bnX), pairW = choose(O, I, T, sms, 0, &bnW);
  if (pairX != pairW) return cudaErrorNotSupported;
  if (pairX) {
    const int g = tileGroup((I + 255) / 256) / 2;
    return fcxGemmBackwardPair(dy, w, x, dx, dw, T, I, O, lddy, ldw, ldx, accumulate, g, g, errFlag, s);
  }
  struct Product {
    CUtensorMap a, b;
    FcxGemmParams p;
    int units, nK;
  };
  auto fill = [&](Product *q, const void *a, const void *b, void *c, int M, int N, int K, int lda, int ldb, int aMN, int bn) {
    if (!(aMN ? makeMap(&q->a, a, K, M, lda, BK) : makeMap(&q->a, a, M, K, lda, BM)) || !makeMap(&q->b, b, K, N, ldb, BK)) return false;
    q->p = FcxGemmParams{};
    q->p.M = M; q->p.N = N; q->p.K = K; q->p.c = c; q->p.ldc = N; q->p.errFlag = errFlag; q->p.bn = bn; q->p.group = tileGroup((N + bn - 1) / bn);
    q->p.aMN = aMN; q->p.bMN = 1;
    q->units = ((M + BM - 1) / BM) * ((N + bn - 1) / bn);
    q->nK = (K + BK - 1) / BK;
    return true;
  };
  Product px, pw;
  if (!fill(&px, dy, w, dx, T, I, O, lddy, ldw, 0, bnX) || !fill(&pw, dy, x, dw, O, I, T, lddy, ldx, 1, bnW)) return cudaErrorNotSupported;
  int swap = 0;
  SecondProduct second{};
  if (!fcxGemmDualPlan(pw.units, pw.nK, fcxGemmPieces(0, O, I, T, pw.units, sms, sms), px.units, px.nK,
                       fcxGemmPieces(0, T, I, O, px.units, sms, sms), sms, &pw.p.splitK, &px.p.splitK, &swap, &second.extra))
    return cudaErrorNotSupported;
  pw.p.accumulate = accumulate;
  int total = 0;
  for (Product *q : {&px, &pw}) {
    total += q->units * q->p.splitK;
    if (q->p.splitK > 1 && !q->p.accumulate) {
      cudaError_t e = cudaMemsetAsync(q->p.c, 0, (size_t)q->p.M * q->p.N * 2, s);
      if (e != cudaSuccess) return e;
    }
  }
  const Product &first = swap ? px : pw, &other = swap ? pw : px;
  second.a = other.a;
  second.b = other.b;
  second.p = other.p;
  FcxDevComm dc{};
  return launch<FCX_GEMM_DUAL>(first.a, first.b, first.p, dc, std::min(total, sms), s, nullptr, &second);
}

// The expert MLP of a mixture-of-experts layer as two grouped GEMMs on CTA pairs (tcgen05.mma.cta_group::2):
//
//   UP    h = silu(x Wg^T) * (x Wu^T)   the activation is computed in the epilogue, from the fp32 accumulators
//   DOWN  y = h Wd^T                    every output row goes straight to the rank and token it belongs to
//
// All local experts run in ONE launch each.  The rows an expert received are a count on the device (the dispatch kernel
// leaves it there); every role of every CTA derives the same tile list from the L counts, so no host round trip and no
// launch per expert is needed, and the tail of one expert's tiles is filled with the next expert's.
//
// A tile is 256 rows (128 per CTA of the pair) x 256 accumulator columns.  UP: the leader CTA loads 128 gate rows of
// the weight and its peer the matching 128 up rows, so both operands of the product lie in the same TMEM lanes, 128
// columns apart, and an epilogue thread needs nobody else's values; the [rows, 2F] intermediate never reaches memory
// (at 16384 rows and F = 14336 that is 0.94 GB written and read again).  Where the tiles are few, a tile is 256 x 128
// columns instead, so that the chain of K steps of a small layer is spread over more SMs; which of the two takes fewer
// waves times the time of a wave (moeTileColumns) depends on the row counts and is decided by every CTA for itself.
//
// Pipeline, barriers and bounded waits are those of the pair kernel in gemm2_sm100.cu.
#include "../kernels/prims.cuh"

#include <algorithm>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_state.h"
#include "moe_gemm_sm100.h"
#include "pdl.cuh"
#include "tcgen05.cuh"

namespace {

using namespace fcxmma;

constexpr int BM = 128, BK = 64, STAGES = 5;
constexpr int A_BYTES = BM * BK * 2;
constexpr int EPI_WARPS = 8, STG_BYTES = 32 * 128;  // staging per epilogue warp: 32 rows x 128 bytes
constexpr int THREADS = 384;

constexpr int BN_MAX = 256, BOX = 64;  // accumulator columns of the wide tile; weight rows per TMA box
constexpr int BOX_BYTES = BOX * BK * 2, STAGE_BYTES = A_BYTES + BN_MAX / 2 * BK * 2;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * STG_BYTES + 1024 + 512;

struct WeightMaps {
  CUtensorMap m[FCX_MOE_MAX_EXPERTS];
};

struct GroupParams {
  int L, capL, N, K;  // N: columns of the result (UP: F, DOWN: H)
  const int *rows;
  int group;
  int *errFlag;
  // DOWN
  const int4 *rowInfo;
  size_t combineOff, doneOff;
  int topk;
};

// 256 or 128 accumulator columns per tile for `rowBlocks` 256-row blocks, `cols` columns and sums of length K.  Narrow tiles
// where they take no more waves.  Otherwise a narrow wave costs about 0.6 to 0.75 of a wide one, which more waves (3 for 2, 5
// for 3, up to twice as many) eat up, except for short sums of the gate / up product, whose wide tiles spend their time on
// the activation.  Measured with cold weights, 8 row blocks, narrow / wide in us.  Gate / up, 3:2 waves: K 256 14.0 / 16.2, 512 15.4 /
// 17.9, 768 17.5 / 19.5, 1024 20.2 / 21.2, 1088 21.1 / 21.6, 1280 23.5 / 23.7, 1536 26.2 / 26.2, 2048 32.9 / 31.7, 3328 47.9 / 44.0; 5:3
// waves: K 256 19.3 / 21.0, 512 21.2 / 22.8, 576 21.7 / 23.2, 768 23.7 / 24.6, 1024 28.4 / 26.6; 2:1 K 1024 15.8 / 15.8, 3328 34.2 / 28.0.
// Down, 3:2: K 512 23.7 / 22.2, 1024 29.8 / 27.4, 2816 52.2 / 45.3, 5632 85.0 / 75.2; 1:1 K 512 18.2 / 18.8, 1024 20.3 / 20.4, 2816 27.1 /
// 29.8.  Both lines could lie a little higher (5:3 up to K 768, 3:2 up to 1280); what that would win is 2 to 6 %.
__host__ __device__ inline int moeTileColumns(long long rowBlocks, int cols, int K, bool up, int pairs) {
  const long long wide = (rowBlocks * ((cols + 255) / 256) + pairs - 1) / pairs, narrow = (rowBlocks * ((cols + 127) / 128) + pairs - 1) / pairs;
  const int tenths = !up || K > 1024 ? 10 : K > 512 ? 15 : 17;  // narrow waves per ten wide ones that still pay
  return narrow * 10 <= wide * tenths ? 128 : 256;
}

template <bool UP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    moeGroupKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmH, const __grid_constant__ WeightMaps wm,
                   const GroupParams p, const FcxDevComm dc) {
  extern __shared__ uint8_t smemRaw[];
  __shared__ int tileStart[FCX_MOE_MAX_EXPERTS + 1];
  __shared__ int rowsOf[FCX_MOE_MAX_EXPERTS];
  __shared__ int tileCols;
  const int warp = warpIndex(), lane = threadIdx.x & 31;
  volatile int *err = p.errFlag;
  const uint32_t cr = ctaRankInCluster();
  const int pair = blockIdx.x >> 1, nPairs = gridDim.x >> 1;

  uint8_t *tiles = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t *epiStage = tiles + STAGES * STAGE_BYTES;
  uint64_t *bars = (uint64_t *)(epiStage + EPI_WARPS * STG_BYTES);
  uint64_t *fullBar = bars, *emptyBar = bars + STAGES, *accFull = bars + 2 * STAGES, *accEmpty = bars + 2 * STAGES + 2;
  uint32_t *tmemBaseSlot = (uint32_t *)(bars + 2 * STAGES + 4);

  const int nK = (p.K + BK - 1) / BK;
  if (threadIdx.x < 64) fcxpdl::pdlWait();  // the row counts come from the kernel before
  if ((int)threadIdx.x < p.L) rowsOf[threadIdx.x] = max(0, min(p.rows[threadIdx.x], p.capL));
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbarInit(&fullBar[s], 1); mbarInit(&emptyBar[s], 1); }
    for (int b = 0; b < 2; b++) { mbarInit(&accFull[b], 1); mbarInit(&accEmpty[b], 2 * EPI_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemBaseSlot)), "r"(2 * BN_MAX) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int blocks = 0, sum = 0;
    for (int e = 0; e < p.L; e++) blocks += (rowsOf[e] + 2 * BM - 1) / (2 * BM);
    const int bnHere = moeTileColumns(blocks, UP ? 2 * p.N : p.N, p.K, UP, nPairs), cols = UP ? bnHere / 2 : bnHere;
    for (int e = 0; e < p.L; e++) {
      tileStart[e] = sum;
      sum += (rowsOf[e] + 2 * BM - 1) / (2 * BM) * ((p.N + cols - 1) / cols);
    }
    tileStart[p.L] = sum;
    tileCols = bnHere;
  }
  fenceBefore();
  __syncthreads();
  clusterSync();  // the peer's barriers exist before anything arrives on them
  fenceAfter();
  const uint32_t tmemBase = *tmemBaseSlot;
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  const int nTiles = tileStart[p.L];
  const int bn = tileCols, bnh = bn / 2, COLS = UP ? bnh : bn;  // COLS: result columns per tile
  const int nN = (p.N + COLS - 1) / COLS;

  // Tile t -> (expert, 256-row block of its segment, column block).  `e` only moves forward: a role's tiles ascend.
  // Inside an expert, bands of `group` row blocks with the row block fastest, as in the plain kernels.
  auto coord = [&](int t, int &e, int *mb, int *nb) {
    while (t >= tileStart[e + 1]) e++;
    const int nM = (rowsOf[e] + 2 * BM - 1) / (2 * BM), u = t - tileStart[e];
    const int perBand = p.group * nN, band = u / perBand, first = band * p.group;
    const int here = min(p.group, nM - first), within = u - band * perBand;
    *mb = first + within % here;
    *nb = within / here;
  };

  if (warp == 0) {
    // ---- TMA producer (both CTAs): own 128 rows of A, own half of the tile's weight rows
    if (electOne()) {
      int stage = 0, e = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < nTiles && ok; t += nPairs) {
        int mb, nb;
        coord(t, e, &mb, &nb);
        const int rowA = e * p.capL + mb * 2 * BM + (int)cr * BM;
        const int rowB = UP ? (int)cr * p.N + nb * bnh : nb * bn + (int)cr * bnh;
        for (int kb = 0; kb < nK; kb++) {
          if (!mbarWait(&emptyBar[stage], phase ^ 1, err)) { ok = false; break; }
          if (cr == 0) mbarExpectTx(&fullBar[stage], 2 * (A_BYTES + bnh * BK * 2));
          const uint32_t bar = mapToCta(smemAddr(&fullBar[stage]), 0);
          uint8_t *sa = tiles + stage * STAGE_BYTES, *sb = sa + A_BYTES;
          tmaLoad2dPair(sa, &tmA, kb * BK, rowA, bar);
          for (int j = 0; j < bnh / BOX; j++) tmaLoad2dPair(sb + j * BOX_BYTES, &wm.m[e], kb * BK, rowB + j * BOX, bar);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one thread of the leader CTA; the warp waits as one
    if (cr == 0) {
      int stage = 0, buf = 0;
      uint32_t phase = 0, accPhase = 0;
      bool ok = true;
      // D fp32, A and B bf16, both K-major, M = 256 over the pair, N = bn
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
      for (int t = pair; t < nTiles && ok; t += nPairs) {
        if (!__all_sync(0xffffffffu, mbarWait(&accEmpty[buf], accPhase ^ 1, err))) break;
        fenceAfter();
        const uint32_t dTmem = tmemBase + (uint32_t)buf * BN_MAX;
        for (int kb = 0; kb < nK; kb++) {
          if (!__all_sync(0xffffffffu, mbarWait(&fullBar[stage], phase, err))) { ok = false; break; }
          fenceAfter();
          if (electOne()) {
            const uint32_t sa = smemAddr(tiles + stage * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / 16; k++)
              mmaF16Pair(dTmem, smemDesc(sa + k * 32), smemDesc(sb + k * 32), idesc, (kb > 0 || k > 0) ? 1u : 0u);
            mmaCommitPair(&emptyBar[stage]);
            if (kb + 1 == nK) mmaCommitPair(&accFull[buf]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (++buf == 2) { buf = 0; accPhase ^= 1; }
      }
    }
  } else if (warp >= 4) {
    // ---- epilogue (both CTAs, 8 warps): warp w owns TMEM lanes [32*(w%4), +32) and the left (warps 4-7) or right
    // (warps 8-11) half of the result columns.  A wait that gives up turns the warp dead: it walks on but touches nothing.
    const int ew = warp - 4, q = ew & 3, half = ew >> 2;
    const int HALF_COLS = COLS / 2;
    int buf = 0, e = 0;
    uint32_t accPhase = 0, chunkNo = 0;
    bool live = true;
    uint8_t *stg = epiStage + (size_t)ew * STG_BYTES;
    for (int t = pair; t < nTiles; t += nPairs) {
      int mb, nb;
      coord(t, e, &mb, &nb);
      if (live) live = __all_sync(0xffffffffu, mbarWait(&accFull[buf], accPhase, err));
      if (live) {
        fenceAfter();
        const int lrow0 = mb * 2 * BM + (int)cr * BM + q * 32, rows = rowsOf[e];  // row inside the expert's segment
        const int col0 = nb * COLS + half * HALF_COLS;
        const uint32_t lanes = tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN_MAX + half * HALF_COLS);
        if (UP) {
          // 32 gate and 32 up columns at a time -> 32 result columns; the TMA unit stores the 32 x 32 block (64-byte
          // swizzle) and clips columns past F.  Rows past the count land in the padding of the expert's own segment
          // (its length is a multiple of 128).
#pragma unroll 1
          for (int c0 = 0; c0 < HALF_COLS; c0 += 32) {
            if (col0 + c0 >= p.N || lrow0 >= rows) break;
            uint32_t g[32], u[32];
            tmemLd32(lanes + c0, g);
            tmemLd32(lanes + bnh + c0, u);
            // two staging blocks of 2 KB: the one about to be refilled must have been read out by the TMA unit
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            __syncwarp();
            tmemLdWait();
#pragma unroll
            for (int j = 0; j < 32; j++) {
              const float gv = __uint_as_float(g[j]);
              g[j] = __float_as_uint(gv / (1.f + __expf(-gv)) * __uint_as_float(u[j]));
            }
            uint4 *blk = (uint4 *)(stg + (chunkNo & 1) * 2048);
#pragma unroll
            for (int v = 0; v < 4; v++) {
              uint4 o;
              o.x = pack2(__uint_as_float(g[8 * v + 0]), __uint_as_float(g[8 * v + 1]));
              o.y = pack2(__uint_as_float(g[8 * v + 2]), __uint_as_float(g[8 * v + 3]));
              o.z = pack2(__uint_as_float(g[8 * v + 4]), __uint_as_float(g[8 * v + 5]));
              o.w = pack2(__uint_as_float(g[8 * v + 6]), __uint_as_float(g[8 * v + 7]));
              blk[lane * 4 + (v ^ ((lane >> 1) & 3))] = o;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                           ::"l"(&tmH), "r"(col0 + c0), "r"(e * p.capL + lrow0), "r"(smemAddr(blk)) : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            chunkNo++;
          }
        } else if (lrow0 < rows) {
          // 64 columns at a time through shared memory (one row per lane in, 8 lanes per 128-byte line out); each lane
          // knows where its row goes, and the lanes that store a line ask it
          char *mine = nullptr;
          if (lrow0 + lane < rows) {
            const int4 info = p.rowInfo[(size_t)e * p.capL + lrow0 + lane];
            mine = dc.heap[info.x] + p.combineOff + ((size_t)info.y * p.topk + info.z) * p.N * 2;
          }
          uint4 *blk = (uint4 *)stg;
#pragma unroll 1
          for (int c0 = 0; c0 < HALF_COLS; c0 += 64) {
            if (col0 + c0 >= p.N) break;
            uint32_t r0[32], r1[32];
            tmemLd32(lanes + c0, r0);
            tmemLd32(lanes + c0 + 32, r1);
            tmemLdWait();
#pragma unroll
            for (int v = 0; v < 8; v++) {
              const uint32_t *r = v < 4 ? r0 + 8 * v : r1 + 8 * (v - 4);
              uint4 o;
              o.x = pack2(__uint_as_float(r[0]), __uint_as_float(r[1]));
              o.y = pack2(__uint_as_float(r[2]), __uint_as_float(r[3]));
              o.z = pack2(__uint_as_float(r[4]), __uint_as_float(r[5]));
              o.w = pack2(__uint_as_float(r[6]), __uint_as_float(r[7]));
              blk[lane * 8 + (v ^ (lane & 7))] = o;
            }
            __syncwarp();
            const int col = col0 + c0 + (lane & 7) * 8;
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const int rr = i * 4 + (lane >> 3);
              char *dst = (char *)__shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)mine, rr);
              const uint4 o = blk[rr * 8 + ((lane & 7) ^ (rr & 7))];
              if (dst && col < p.N) *(uint4 *)(dst + (size_t)col * 2) = o;  // N is a multiple of 8
            }
            __syncwarp();
          }
        }
        fenceBefore();
        __syncwarp();
        if (lane == 0) mbarArriveRemote(mapToCta(smemAddr(&accEmpty[buf]), 0));
      }
      if (++buf == 2) { buf = 0; accPhase ^= 1; }
    }
    if (UP && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  // ---- tear-down: nobody leaves, and no TMEM is freed, while the peer may still use this CTA's memory or barriers
  fenceBefore();
  __syncthreads();
  clusterSync();
  fenceAfter();
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(2 * BN_MAX) : "memory");
  if (!UP) {
    // every row this CTA produced has been stored (possibly on peers): tell every rank that this CTA is done
    __threadfence_system();
    __syncthreads();
    if ((int)threadIdx.x < dc.nranks) {
      uint64_t *cnt = (uint64_t *)(dc.heap[threadIdx.x] + p.doneOff);
      asm volatile("red.release.sys.global.add.u64 [%0], %1;" ::"l"(cnt), "l"((uint64_t)1) : "memory");
    }
  }
}

int pairCount() { return fcxhost::smCount() / 2; }

template <bool UP>
cudaError_t launchGroup(const CUtensorMap &a, const CUtensorMap &h, const WeightMaps &wm, const GroupParams &p, const FcxDevComm &dc,
                        cudaStream_t s) {
  static fcxhost::OncePerDevice once;
  const cudaError_t e = once([] { return cudaFuncSetAttribute(moeGroupKernel<UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES); });
  if (e != cudaSuccess) return e;
  return fcxpdl::launchPdl(moeGroupKernel<UP>, 2 * pairCount(), THREADS, SMEM_BYTES, s, a, h, wm, p, dc);
}

}  // namespace

extern "C" int fcxMoeTileColumns(int rowBlocks, int cols, int K, int up, int pairs) { return moeTileColumns(rowBlocks, cols, K, up != 0, pairs); }

extern "C" cudaError_t fcxMoeUpGrouped(const void *x, const void *const *w, void *h, const int *rows, int L, int capL, int H, int F,
                                       const int *ldw, int *errFlag, cudaStream_t s) {
  if (L < 1 || L > FCX_MOE_MAX_EXPERTS || capL <= 0 || capL % 128 || H % 8 || F % 8 || H <= 0 || F <= 0) return cudaErrorInvalidValue;
  if (((uintptr_t)x | (uintptr_t)h) & 15) return cudaErrorInvalidValue;
  CUtensorMap ma, mh;
  WeightMaps wm{};
  if (!makeTileMap(&ma, x, (uint64_t)L * capL, H, H, BM, 2) || !makeStoreMap(&mh, h, (uint64_t)L * capL, F, F)) return cudaErrorNotSupported;
  for (int e = 0; e < L; e++)
    if (ldw[e] % 8 || ((uintptr_t)w[e] & 15) || !makeTileMap(&wm.m[e], w[e], 2 * (uint64_t)F, H, ldw[e], BOX, 2))
      return cudaErrorInvalidValue;
  GroupParams p{};
  p.L = L; p.capL = capL; p.N = F; p.K = H; p.rows = rows; p.group = 8; p.errFlag = errFlag;
  FcxDevComm dc{};
  return launchGroup<true>(ma, mh, wm, p, dc, s);
}

extern "C" cudaError_t fcxMoeDownGrouped(const FcxDevComm *dc, const void *h, const void *const *w, const int *rows, int L, int capL, int H,
                                         int F, int ldh, const int *ldw, const void *rowInfo, size_t combineOff, size_t doneOff, int topk,
                                         int *errFlag, int *gridOut, cudaStream_t s) {
  if (L < 1 || L > FCX_MOE_MAX_EXPERTS || capL <= 0 || H % 8 || F % 8 || H <= 0 || F <= 0 || ldh % 8) return cudaErrorInvalidValue;
  if ((uintptr_t)h & 15) return cudaErrorInvalidValue;
  CUtensorMap ma;
  WeightMaps wm{};
  if (!makeTileMap(&ma, h, (uint64_t)L * capL, F, ldh, BM, 2)) return cudaErrorNotSupported;
  for (int e = 0; e < L; e++)
    if (ldw[e] % 8 || ((uintptr_t)w[e] & 15) || !makeTileMap(&wm.m[e], w[e], H, F, ldw[e], BOX, 2)) return cudaErrorInvalidValue;
  GroupParams p{};
  p.L = L; p.capL = capL; p.N = H; p.K = F; p.rows = rows; p.group = 8; p.errFlag = errFlag;
  p.rowInfo = (const int4 *)rowInfo; p.combineOff = combineOff; p.doneOff = doneOff; p.topk = topk;
  if (gridOut) *gridOut = 2 * pairCount();  // the receivers count one arrival per CTA of every rank
  return launchGroup<false>(ma, ma, wm, p, *dc, s);
}

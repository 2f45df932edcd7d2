// Block-scaled fp8 (e4m3) GEMM on tcgen05: C[M,N] (bf16) = (A_q * sa) x (B_q * sb)^T.
//
// Scaling granularity is the one used for fp8 training of large transformer
// layers: activations carry one fp32 scale per row and 128 columns of K
// (sa[K/128][M]), weights one per 128x128 block (sb[ceil(N/128)][K/128]).
// The tensor cores cannot apply such scales themselves, so every 128-deep
// slice of K is multiplied into a TMEM accumulator of its own (tcgen05.mma
// kind::f8f6f4, fp32 accumulate) and the epilogue warps fold it into
// registers as acc += sa[row,kb] * sb[nb,kb] * partial while the next slices
// are already being multiplied.
//
// The reference has no GEMM; its users would pair flagcx collectives with a
// vendor scaled matmul.
//
// Two kernels, persistent over their tiles:
//   gemmFp8PairKernel  256 x 256 tiles on CTA pairs (cta_group::2), two 256-column accumulators.  A CTA fetches 32 KB per
//                      slice for 128 x 256 results; the 128 x 128 tiles of the one-CTA kernel fetch the same for half of
//                      them, and L2 cannot deliver that to 148 SMs at the fp8 rate.
//   gemmFp8Kernel<BN>  128 x BN tiles on single CTAs (BN 128 or 64), four accumulators: for outputs with too few tiles; with fewer
//                      still, the two or four CTAs of a cluster share a tile, a stretch of K each.
// Roles: warps 0-7 promotion + epilogue (warp w reads TMEM lanes 32*(w%4).., one output row per thread, and half of the
// tile's columns), warp 8 TMA producer (128-byte swizzle, no multicast), warp 9 MMA issuer and TMEM allocation.
// The single-CTA kernel commits ONCE per slice, on the barrier of the slice's stage: the producer and the epilogue both wait for it.
// It has at least as many stages as accumulators, so that neither can miss a phase: the stage is not refilled before the producer
// has seen it done, nor its successor multiplied before the epilogue has freed the accumulator.  On CTA pairs one commit was no
// faster.
// Every wait is bounded; a wait that gives up sets the error flag and the kernel drains and returns.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_state.h"
#include "gemm_fp8_sm100.h"
#include "pdl.cuh"
#include "tcgen05.cuh"

namespace {

using namespace fcxmma;

constexpr int BM = 128, BK = 128;
constexpr int A_BYTES = BM * BK;
constexpr int EPI_WARPS = 8, THREADS = 320;
constexpr int STG_BYTES = 32 * 64;  // a block of 32 rows x 32 bf16 columns on its way to the TMA unit; two per epilogue warp
constexpr int EPI_BYTES = EPI_WARPS * 2 * STG_BYTES;

struct Params {
  int M, N, K;
  const float *sa;  // [K/128][M]
  const float *sb;  // [ceil(N/128)][K/128]
  int group;
  int *errFlag;
};

// D fp32, A and B e4m3 (format 0), both K-major
__device__ __forceinline__ constexpr uint32_t instrDescF8(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }

__device__ __forceinline__ void tileCoord(const Params &p, int nM, int nN, int t, int *mb, int *nb) {
  const int perBand = p.group * nN, band = t / perBand, first = band * p.group;
  const int rowsHere = min(p.group, nM - first), within = t - band * perBand;
  *mb = first + within % rowsHere;
  *nb = within / rowsHere;
}

// The scales of one output row, GROUP slices at a time.  The loads of the next group are issued together when a group
// begins and used when it ends: a load per slice, even one issued eight slices ahead, made every slice wait for the
// youngest outstanding load (about 800 clocks a slice in place of the 256 its multiplication takes).
template <int GROUP>
struct Scales {
  const float *a, *b;
  int M, nK;
  float cur[GROUP], na[GROUP], nb[GROUP];
  __device__ __forceinline__ void fetch(int kb0) {
#pragma unroll
    for (int j = 0; j < GROUP; j++) {
      na[j] = kb0 + j < nK ? a[(size_t)(kb0 + j) * M] : 0.f;
      nb[j] = kb0 + j < nK ? b[kb0 + j] : 0.f;
    }
  }
  __device__ __forceinline__ void turn() {
#pragma unroll
    for (int j = 0; j < GROUP; j++) cur[j] = na[j] * nb[j];
  }
};

// On CTA pairs: the scales of the slices in flight, a ring in shared memory that the producer warp fills with 4-byte cp.async, so that no
// thread ever waits for a load of its own.  A slot holds the activation scales of the CTA's 128 rows and the weight scales of
// the tile's column blocks.  RING = stages + accumulators slots need no barrier of their own to be free: the slot of slice j is
// filled once the stage of slice j - stages has been multiplied, which began after every epilogue warp was done with slice
// j - stages - accumulators.  (Held in registers, a group of four slices ahead, they did not fit beside 128 sums a thread, and every
// group stalled for 1300 clocks: 8192 x 4096 x 4096 took 142 us and takes 126, 8192 x 1024 x 4096 47.8 and 39.4.  The single-CTA
// kernels have the room: there the ring is a wait more per slice, 333 x 1792 x 4096 12.5 us with registers and 12.9 with it.)
struct ScaleSlot {
  float a[BM];
  float b[2];
  float pad[2];
};
__device__ __forceinline__ void cpAsync4(void *smemDst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smemAddr(smemDst)), "l"(src) : "memory");
}
// All lanes of the producer warp: rows row0 .. +127 (clamped to the matrix), column blocks `block` .. + BLOCKS - 1, slice kb.
template <int BLOCKS>
__device__ __forceinline__ void fetchScales(ScaleSlot *slot, uint64_t *bar, const Params &p, int row0, int block, int kb, int nK, int lane) {
  const float *a = p.sa + (size_t)kb * p.M;
#pragma unroll
  for (int i = 0; i < BM / 32; i++) cpAsync4(&slot->a[i * 32 + lane], a + min(row0 + i * 32 + lane, p.M - 1));
  if (lane < BLOCKS) cpAsync4(&slot->b[lane], p.sb + (size_t)min(block + lane, (p.N - 1) / 128) * nK + kb);
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smemAddr(bar)) : "memory");
}

// COLS fp32 values per lane (one row) -> bf16 -> C, 32 columns at a time through this warp's two staging blocks (laid out
// as the TMA unit's 64-byte swizzle wants them); the unit clips what lies beyond M and N.
template <int COLS>
__device__ __forceinline__ void storeRows(const float (&acc)[COLS], const CUtensorMap *tmC, uint8_t *stg, int row0, int col0, int M, int N, int lane,
                                          uint32_t *blockNo) {
#pragma unroll
  for (int c0 = 0; c0 < COLS; c0 += 32) {
    if (row0 < M && col0 + c0 < N) {
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      __syncwarp();
      uint4 *blk = (uint4 *)(stg + (*blockNo & 1) * STG_BYTES);  // the one whose store is the older
      ++*blockNo;
#pragma unroll
      for (int v = 0; v < 4; v++) {
        uint4 o;
        o.x = pack2(acc[c0 + 8 * v + 0], acc[c0 + 8 * v + 1]);
        o.y = pack2(acc[c0 + 8 * v + 2], acc[c0 + 8 * v + 3]);
        o.z = pack2(acc[c0 + 8 * v + 4], acc[c0 + 8 * v + 5]);
        o.w = pack2(acc[c0 + 8 * v + 6], acc[c0 + 8 * v + 7]);
        blk[lane * 4 + (v ^ ((lane >> 1) & 3))] = o;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];"
                     ::"l"(tmC), "r"(col0 + c0), "r"(row0), "r"(smemAddr(blk)) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
  }
}

// ------------------------------------------------------------------ one CTA per tile

constexpr int stageBytes(int bn) { return A_BYTES + bn * BK; }
constexpr int stages(int bn) { return bn == 128 ? 5 : 7; }
constexpr int smemBytes(int bn) { return stages(bn) * stageBytes(bn) + EPI_BYTES + 1024 + 256; }

template <int BN, bool CUT>
__global__ void __launch_bounds__(THREADS, 1) gemmFp8Kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                                                            const __grid_constant__ CUtensorMap tmC, const Params p) {
  constexpr int STAGES = stages(BN), STAGE_BYTES = stageBytes(BN), ACC_BUFS = 4, COLS = BN / 2;
  extern __shared__ uint8_t smemRaw[];
  const int warp = warpIndex(), lane = threadIdx.x & 31;
  volatile int *err = p.errFlag;
  uint8_t *tiles = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t *epiStage = tiles + STAGES * STAGE_BYTES;
  uint64_t *bars = (uint64_t *)(epiStage + EPI_BYTES);
  uint64_t *fullBar = bars, *doneBar = bars + STAGES, *tmemEmpty = bars + 2 * STAGES;
  uint32_t *tmemBaseSlot = (uint32_t *)(bars + 2 * STAGES + ACC_BUFS);

  const int nN = (p.N + BN - 1) / BN, nM = (p.M + BM - 1) / BM, nTiles = nN * nM, nKAll = p.K / BK;
  // CUT: the CTAs of a cluster share a tile, each with its own stretch of K; a tile per cluster
  const int split = CUT ? (int)gridDim.x / nTiles : 1, rank = CUT ? (int)ctaRankInCluster() : 0, per = (nKAll + split - 1) / split;
  const int kLo = rank * per, nK = min(nKAll, kLo + per), tile0 = CUT ? (int)blockIdx.x / split : (int)blockIdx.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbarInit(&fullBar[s], 1); mbarInit(&doneBar[s], 1); }
    for (int b = 0; b < ACC_BUFS; b++) mbarInit(&tmemEmpty[b], EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemBaseSlot)), "r"(ACC_BUFS * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fenceBefore();
  __syncthreads();
  fenceAfter();
  const uint32_t tmemBase = *tmemBaseSlot;
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();  // everything above touches only this CTA's own memories

  if (warp == 8) {
    if (electOne()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = tile0; t < nTiles && ok; t += gridDim.x) {
        int mb, nb;
        tileCoord(p, nM, nN, t, &mb, &nb);
        for (int kb = kLo; kb < nK; kb++) {
          if (!mbarWait(&doneBar[stage], phase ^ 1, err)) { ok = false; break; }
          mbarExpectTx(&fullBar[stage], STAGE_BYTES);
          uint8_t *sa = tiles + stage * STAGE_BYTES, *sb = sa + A_BYTES;
          tmaLoad2d(sa, &tmA, kb * BK, mb * BM, &fullBar[stage]);
          tmaLoad2d(sb, &tmB, kb * BK, nb * BN, &fullBar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
    if (CUT) { clusterSync(); clusterSync(); }
  } else if (warp == 9) {  // the warp waits as one, one lane issues
    int stage = 0, buf = 0;
    uint32_t phase = 0, accPhase = 0;
    bool ok = true;
    const uint32_t idesc = instrDescF8(BM, BN);
    for (int t = tile0; t < nTiles && ok; t += gridDim.x) {
      for (int kb = kLo; kb < nK; kb++) {
        if (!__all_sync(0xffffffffu, mbarWait(&tmemEmpty[buf], accPhase ^ 1, err) && mbarWait(&fullBar[stage], phase, err))) { ok = false; break; }
        fenceAfter();
        if (electOne()) {
          const uint32_t dTmem = tmemBase + (uint32_t)buf * BN;
          const uint32_t sa = smemAddr(tiles + stage * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 32; k++)  // 32 fp8 = 32 bytes further along K inside the 128-byte swizzle row
            mmaF8(dTmem, smemDesc(sa + k * 32), smemDesc(sb + k * 32), idesc, k > 0 ? 1u : 0u);
          mmaCommit(&doneBar[stage]);  // the stage may be refilled and the accumulator read
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        if (++buf == ACC_BUFS) { buf = 0; accPhase ^= 1; }
      }
    }
    if (CUT) { clusterSync(); clusterSync(); }
  } else {
    const int q = warp & 3, half = warp >> 2;  // TMEM lane quarter (fixed by warp index % 4) and column half
    constexpr int GROUP = 8;
    int buf = 0, stage = 0;
    uint32_t phase = 0, blockNo = 0;
    bool live = true;
    uint8_t *stg = epiStage + (size_t)warp * 2 * STG_BYTES;
    for (int t = tile0; t < nTiles; t += gridDim.x) {
      int mb, nb;
      tileCoord(p, nM, nN, t, &mb, &nb);
      const int row0 = mb * BM + q * 32;
      Scales<GROUP> sc{p.sa + min(row0 + lane, p.M - 1), p.sb + (size_t)(nb * BN / 128) * nKAll, p.M, nK};
      sc.fetch(kLo);
      float acc[COLS];
#pragma unroll
      for (int j = 0; j < COLS; j++) acc[j] = 0.f;
      sc.turn();
      for (int kb0 = kLo; kb0 < nK; kb0 += GROUP) {
        sc.fetch(kb0 + GROUP);
#pragma unroll
        for (int j = 0; j < GROUP; j++) {
          if (kb0 + j < nK) {
            if (live) live = __all_sync(0xffffffffu, mbarWait(&doneBar[stage], phase, err));
            if (live) {
              fenceAfter();
              uint32_t r[COLS];
              const uint32_t taddr = tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + half * COLS);
#pragma unroll
              for (int c = 0; c < COLS; c += 32) tmemLd32(taddr + c, r + c);
              tmemLdWait();
              fenceBefore();
              __syncwarp();
              if (lane == 0) mbarArrive(&tmemEmpty[buf]);  // the values are in registers: the accumulator may be overwritten
#pragma unroll
              for (int i = 0; i < COLS; i++) acc[i] = fmaf(sc.cur[j], __uint_as_float(r[i]), acc[i]);
            }
            if (++buf == ACC_BUFS) buf = 0;
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        }
        sc.turn();
      }
      if (CUT) {
        // Every CTA finishes an equal share of the tile's (32 rows x COLS columns) pieces, one per warp: `owner` of this warp's.  The
        // others send it their sums, a row of 32 lanes per column, into the stages' memory, which is free once every CTA of the
        // cluster has multiplied its last slice; they are added in the order of K.
        const int share = EPI_WARPS / split, owner = split == 2 ? half : half + 2 * (q >> 1), mine = split == 2 ? q : q & 1;
        auto place = [&](int from) { return (float *)tiles + ((size_t)(from - (from > owner)) * share + mine) * COLS * 32 + lane; };
        clusterSync();
        if (rank != owner) {
          const uint32_t to = mapToCta(smemAddr(place(rank)), owner);
#pragma unroll
          for (int j = 0; j < COLS; j++) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + j * 128), "f"(acc[j]) : "memory");
        }
        clusterSync();
        if (rank != owner) break;
        for (int r = 1; r < split; r++) {
          const float *got = place(r <= owner ? r - 1 : r);
#pragma unroll
          for (int j = 0; j < COLS; j++) acc[j] += got[j * 32];
        }
      }
      if (live) storeRows<COLS>(acc, &tmC, stg, row0, nb * BN + half * COLS, p.M, p.N, lane, &blockNo);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  fenceBefore();
  __syncthreads();
  fenceAfter();
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(ACC_BUFS * BN) : "memory");
}

// ------------------------------------------------------------------ CTA pairs, 256 x 256 tiles

constexpr int PN = 256, PNH = 128, PSTAGES = 5, PSTAGE_BYTES = A_BYTES + PNH * BK, PRING = PSTAGES + 2;
constexpr int PTHREADS = 384;  // three warp groups: two of epilogue warps, one for the producer and the issuer
// 128 sums per thread need more than the 168 registers that 384 threads get each: the third group gives some of its own.
// 216 x 256 + 72 x 128 = 168 x 384.
constexpr int EPI_REGS = 216, ROLE_REGS = 72;
constexpr int PSMEM_BYTES = PSTAGES * PSTAGE_BYTES + EPI_BYTES + PRING * (int)sizeof(ScaleSlot) + 1024 + 256;
static_assert(PSMEM_BYTES <= 232448, "shared memory of one CTA");

__device__ __forceinline__ void mmaF8Pair(uint32_t dTmem, uint64_t aDesc, uint64_t bDesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(dTmem), "l"(aDesc), "l"(bDesc), "r"(idesc), "r"(accumulate) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PTHREADS, 1)
    gemmFp8PairKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                      const Params p) {
  extern __shared__ uint8_t smemRaw[];
  const int warp = warpIndex(), lane = threadIdx.x & 31;
  volatile int *err = p.errFlag;
  const uint32_t cr = ctaRankInCluster();  // 0 = leader
  const int pair = blockIdx.x >> 1, nPairs = gridDim.x >> 1;
  uint8_t *tiles = (uint8_t *)(((uintptr_t)smemRaw + 1023) & ~(uintptr_t)1023);
  uint8_t *epiStage = tiles + PSTAGES * PSTAGE_BYTES;
  ScaleSlot *scales = (ScaleSlot *)(epiStage + EPI_BYTES);
  uint64_t *bars = (uint64_t *)(scales + PRING);
  uint64_t *fullBar = bars, *emptyBar = bars + PSTAGES, *accFull = bars + 2 * PSTAGES, *accEmpty = accFull + 2, *scaleFull = accEmpty + 2;
  uint32_t *tmemBaseSlot = (uint32_t *)(scaleFull + PRING);

  const int nN = (p.N + PN - 1) / PN, nM = (p.M + 2 * BM - 1) / (2 * BM), nTiles = nN * nM, nK = p.K / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < PSTAGES; s++) { mbarInit(&fullBar[s], 1); mbarInit(&emptyBar[s], 1); }
    for (int b = 0; b < 2; b++) { mbarInit(&accFull[b], 1); mbarInit(&accEmpty[b], 2 * EPI_WARPS); }  // the warps of both CTAs
    for (int r = 0; r < PRING; r++) mbarInit(&scaleFull[r], 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tmemBaseSlot)), "r"(2 * PN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fenceBefore();
  __syncthreads();
  clusterSync();  // the peer's barriers exist before anything arrives on them
  fenceAfter();
  const uint32_t tmemBase = *tmemBaseSlot;
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();  // everything above touches only this CTA's own memories

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ROLE_REGS));
    if (warp == 8) {
      // ---- TMA producer (both CTAs): own 128 rows of A, own 128 of the 256 weight rows, bytes counted on the leader's barrier;
      // and the scales of its own rows, on its own barrier
      int stage = 0, slot = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < nTiles && ok; t += nPairs) {
        int mb, nb;
        tileCoord(p, nM, nN, t, &mb, &nb);
        const int row0 = mb * 2 * BM + (int)cr * BM;
        for (int kb = 0; kb < nK; kb++) {
          if (!__all_sync(0xffffffffu, mbarWait(&emptyBar[stage], phase ^ 1, err))) { ok = false; break; }
          if (electOne()) {
            if (cr == 0) mbarExpectTx(&fullBar[stage], 2 * PSTAGE_BYTES);
            const uint32_t bar = mapToCta(smemAddr(&fullBar[stage]), 0);
            uint8_t *sa = tiles + stage * PSTAGE_BYTES, *sb = sa + A_BYTES;
            tmaLoad2dPair(sa, &tmA, kb * BK, row0, bar);
            tmaLoad2dPair(sb, &tmB, kb * BK, nb * PN + (int)cr * PNH, bar);
          }
          __syncwarp();
          fetchScales<2>(&scales[slot], &scaleFull[slot], p, row0, nb * 2, kb, nK, lane);
          if (++stage == PSTAGES) { stage = 0; phase ^= 1; }
          if (++slot == PRING) slot = 0;
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 9) {
      // ---- MMA issuer: one thread of the leader CTA; the warp waits as one
      if (cr == 0) {
        int stage = 0, buf = 0;
        uint32_t phase = 0, accPhase = 0;
        bool ok = true;
        const uint32_t idesc = instrDescF8(2 * BM, PN);
        for (int t = pair; t < nTiles && ok; t += nPairs) {
          for (int kb = 0; kb < nK; kb++) {
            if (!__all_sync(0xffffffffu, mbarWait(&fullBar[stage], phase, err) && mbarWait(&accEmpty[buf], accPhase ^ 1, err))) { ok = false; break; }
            fenceAfter();
            if (electOne()) {
              const uint32_t sa = smemAddr(tiles + stage * PSTAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
              for (int k = 0; k < BK / 32; k++)
                mmaF8Pair(tmemBase + (uint32_t)buf * PN, smemDesc(sa + k * 32), smemDesc(sb + k * 32), idesc, k > 0 ? 1u : 0u);
              mmaCommitPair(&emptyBar[stage]);
              mmaCommitPair(&accFull[buf]);
            }
            __syncwarp();
            if (++stage == PSTAGES) { stage = 0; phase ^= 1; }
            if (++buf == 2) { buf = 0; accPhase ^= 1; }
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
    // ---- promotion + epilogue (both CTAs): 128 fp32 sums per thread.  A warp's 128 columns are one scale block of the weight.
    const int q = warp & 3, half = warp >> 2;
    constexpr int COLS = 128;
    int buf = 0, slot = 0;
    uint32_t accPhase = 0, scalePhase = 0, blockNo = 0;
    bool live = true;
    uint8_t *stg = epiStage + (size_t)warp * 2 * STG_BYTES;
    const uint32_t emptyAddr = mapToCta(smemAddr(accEmpty), 0);
    const uint32_t lanes = tmemBase + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * COLS);
    for (int t = pair; t < nTiles; t += nPairs) {
      int mb, nb;
      tileCoord(p, nM, nN, t, &mb, &nb);
      float acc[COLS];
#pragma unroll
      for (int j = 0; j < COLS; j++) acc[j] = 0.f;
#pragma unroll 1
      for (int kb = 0; kb < nK && live; kb++) {
        live = __all_sync(0xffffffffu, mbarWait(&scaleFull[slot], scalePhase, err));
        const float sc = scales[slot].a[q * 32 + lane] * scales[slot].b[half];
        if (live) live = __all_sync(0xffffffffu, mbarWait(&accFull[buf], accPhase, err));
        if (live) {
          fenceAfter();
#pragma unroll
          for (int c = 0; c < COLS; c += 32) {
            uint32_t r[32];
            tmemLd32(lanes + buf * PN + c, r);
            tmemLdWait();
            if (c + 32 == COLS) {
              fenceBefore();
              __syncwarp();
              if (lane == 0) mbarArriveRemote(emptyAddr + buf * 8);  // all of it is in registers
            }
#pragma unroll
            for (int i = 0; i < 32; i++) acc[c + i] = fmaf(sc, __uint_as_float(r[i]), acc[c + i]);
          }
        }
        if (++buf == 2) { buf = 0; accPhase ^= 1; }
        if (++slot == PRING) { slot = 0; scalePhase ^= 1; }
      }
      if (live) storeRows<COLS>(acc, &tmC, stg, mb * 2 * BM + (int)cr * BM + q * 32, nb * PN + half * COLS, p.M, p.N, lane, &blockNo);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  // ---- tear-down: nobody leaves, and no TMEM is freed, while the peer may still use this CTA's memory or barriers
  fenceBefore();
  __syncthreads();
  clusterSync();
  fenceAfter();
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(2 * PN) : "memory");
}

// ------------------------------------------------------------------ quantisation

// Four fp32 values -> four e4m3 bytes.
__device__ __forceinline__ uint32_t pack4Fp8(float a, float b, float c, float d) {
  return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3) |
         (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3) << 16;
}

// scale = amax / 448 over a (row, 128-column block), q = x / scale.  A lane holds VEC consecutive values (8: half a warp
// per block, 16-byte loads; 4: a warp per block, for rows that are only 8-byte aligned) of UNROLL blocks whose loads are
// all issued before the first is used: one 8-byte load in flight per lane left the kernel waiting (2.1 TB/s).
template <int VEC, int UNROLL>
__global__ void __launch_bounds__(256) quantActKernel(const __nv_bfloat16 *x, __nv_fp8_storage_t *q, float *sa, int M, int K, int ldx) {
  constexpr int LANES = 128 / VEC, PER_CTA = 256 / LANES;  // lanes per block, blocks per CTA and step
  const uint32_t nKb = K / 128;
  const uint64_t total = (uint64_t)M * nKb;
  const int sub = threadIdx.x / LANES, l = threadIdx.x % LANES;
  const uint64_t first = (uint64_t)blockIdx.x * PER_CTA * UNROLL + sub;
  // One division for the first block, additions for the others: a 64-bit division and remainder for every block, once to
  // load and once to store it, took longer than the loads (39 us in place of 23 at 8192 x 4096, 101 MB).
  uint32_t row0, kb0;
  if (total <= 0xffffffffu) {
    row0 = (uint32_t)first / nKb;
    kb0 = (uint32_t)first - row0 * nKb;
  } else {
    row0 = (uint32_t)(first / nKb);
    kb0 = (uint32_t)(first - (uint64_t)row0 * nKb);
  }
  const uint32_t rowStep = PER_CTA / nKb, kbStep = PER_CTA - rowStep * nKb;
  uint32_t rows[UNROLL], kbs[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; u++) {
    rows[u] = row0;
    kbs[u] = kb0;
    row0 += rowStep;
    kb0 += kbStep;
    if (kb0 >= nKb) { kb0 -= nKb; row0++; }
  }
  fcxpdl::pdlRelease();
  fcxpdl::pdlWait();
  uint32_t raw[UNROLL][VEC / 2];
#pragma unroll
  for (int u = 0; u < UNROLL; u++) {
    if (first + (uint64_t)u * PER_CTA < total) {
      const __nv_bfloat16 *src = x + (size_t)rows[u] * ldx + kbs[u] * 128 + l * VEC;
      if (VEC == 8) *(uint4 *)raw[u] = *(const uint4 *)src;
      else *(uint2 *)raw[u] = *(const uint2 *)src;
    } else {
#pragma unroll
      for (int j = 0; j < VEC / 2; j++) raw[u][j] = 0;
    }
  }
#pragma unroll
  for (int u = 0; u < UNROLL; u++) {
    float v[VEC], amax = 0.f;
#pragma unroll
    for (int j = 0; j < VEC / 2; j++) {
      const float2 f = __bfloat1622float2(*(const __nv_bfloat162 *)&raw[u][j]);
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
      amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (first + (uint64_t)u * PER_CTA >= total) continue;
    const float scale = amax > 0.f ? amax / 448.f : 1.f, inv = 1.f / scale;
    uint32_t out[VEC / 4];
#pragma unroll
    for (int j = 0; j < VEC / 4; j++) out[j] = pack4Fp8(v[4 * j] * inv, v[4 * j + 1] * inv, v[4 * j + 2] * inv, v[4 * j + 3] * inv);
    __nv_fp8_storage_t *dst = q + (size_t)rows[u] * K + kbs[u] * 128 + l * VEC;
    if (VEC == 8) *(uint2 *)dst = make_uint2(out[0], out[VEC / 4 - 1]);
    else *(uint32_t *)dst = out[0];
    if (l == 0) sa[(size_t)kbs[u] * M + rows[u]] = scale;
  }
}

// One CTA per 128x128 block of the weight.
__global__ void __launch_bounds__(256) quantWeightKernel(const __nv_bfloat16 *__restrict__ w, __nv_fp8_storage_t *__restrict__ q,
                                                         float *__restrict__ sb, int N, int K, int ldw) {
  const int nKb = K / 128, nb = blockIdx.x / nKb, kb = blockIdx.x % nKb;
  __shared__ float red[8];
  __shared__ float scaleS;
  // thread -> (row offset, 4 columns): 32 lanes cover 128 columns, 8 warps step through the rows
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float amax = 0.f;
  for (int r = warp; r < 128; r += 8) {
    const int row = nb * 128 + r;
    if (row < N) {
      const uint2 raw = *(const uint2 *)(w + (size_t)row * ldw + kb * 128 + lane * 4);
      const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw;
      float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = 0.f;
    for (int i = 0; i < 8; i++) m = fmaxf(m, red[i]);
    scaleS = m > 0.f ? m / 448.f : 1.f;
    sb[(size_t)nb * nKb + kb] = scaleS;
  }
  __syncthreads();
  const float inv = 1.f / scaleS;
  for (int r = warp; r < 128; r += 8) {
    const int row = nb * 128 + r;
    if (row < N) {
      const uint2 raw = *(const uint2 *)(w + (size_t)row * ldw + kb * 128 + lane * 4);
      const __nv_bfloat162 *h = (const __nv_bfloat162 *)&raw;
      float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
      uint32_t out = (uint32_t)__nv_cvt_float_to_fp8(a.x * inv, __NV_SATFINITE, __NV_E4M3) |
                     (uint32_t)__nv_cvt_float_to_fp8(a.y * inv, __NV_SATFINITE, __NV_E4M3) << 8 |
                     (uint32_t)__nv_cvt_float_to_fp8(b.x * inv, __NV_SATFINITE, __NV_E4M3) << 16 |
                     (uint32_t)__nv_cvt_float_to_fp8(b.y * inv, __NV_SATFINITE, __NV_E4M3) << 24;
      *(uint32_t *)(q + (size_t)row * K + kb * 128 + lane * 4) = out;
    }
  }
}

using fcxhost::smCount;

}  // namespace

namespace {

template <int BN, bool CUT>
cudaError_t launchOne(const CUtensorMap &ma, const void *bq, const CUtensorMap &mc, const Params &p, int cut, cudaStream_t s) {
  CUtensorMap mb;
  if (!makeTileMap(&mb, bq, p.N, p.K, p.K, BN, 1)) return cudaErrorNotSupported;
  static fcxhost::OncePerDevice once;
  const cudaError_t e = once([] { return cudaFuncSetAttribute(gemmFp8Kernel<BN, CUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes(BN)); });
  if (e != cudaSuccess) return e;
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  if (CUT) return fcxpdl::launchPdlAttr(gemmFp8Kernel<BN, CUT>, tiles * cut, THREADS, smemBytes(BN), dim3(cut, 1, 1), s, ma, mb, mc, p);
  return fcxpdl::launchPdl(gemmFp8Kernel<BN, CUT>, std::min(tiles, smCount()), THREADS, smemBytes(BN), s, ma, mb, mc, p);
}

cudaError_t launchPair(const CUtensorMap &ma, const void *bq, const CUtensorMap &mc, const Params &p, cudaStream_t s) {
  CUtensorMap mb;
  if (!makeTileMap(&mb, bq, p.N, p.K, p.K, PNH, 1)) return cudaErrorNotSupported;
  static fcxhost::OncePerDevice once;
  const cudaError_t e = once([] { return cudaFuncSetAttribute(gemmFp8PairKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PSMEM_BYTES); });
  if (e != cudaSuccess) return e;
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + PN - 1) / PN);
  return fcxpdl::launchPdl(gemmFp8PairKernel, 2 * std::min(tiles, smCount() / 2), PTHREADS, PSMEM_BYTES, s, ma, mb, mc, p);
}

}  // namespace

// Which tile: 0 = 256 x 256 on CTA pairs, 128 or 64 = 128 x that many columns on single CTAs; and how many CTAs of a cluster share
// one, each with a stretch of K.  The time is about the number of waves times the time of the 128-deep slices of a tile, in
// nanoseconds; with more than one wave the single CTAs' slices get longer (L2), and the tiles follow one another with a gap, which is what
// short sums consist of.  Measured, us for pairs / 128 / 64 columns, K whole:
// 8192 x 1024 x 4096 39.0 / 47.2 / 69.1, 4096 x 4096 x 1024 25.9 / 27.5 / 39.2, 3000 x 2000 x 4096 37.5 / 36.4 / 58.9, 1024 x 4096 x 2048
// 13.3 / 14.9 / 22.6, 512 x 4096 x 4096 20.7 / 14.3 / 22.1, 1024 x 1024 x 1024 8.5 / 6.1 / 5.5, 333 x 1792 x 4096 19.8 / 13.4 / 12.5.
// 8192 x 4096 x 128 15.7 / 24.2 / 36.1, x 512 27.0 / 33.5 / 49.6, x 1024 39.9 / 47.8 / 73.0, 2048 x 2048 x 128 5.5 / 5.1 / 6.9.
// Cut in 2 or 4 as long as all clusters fit on the chip at once; it costs two barriers of the cluster and the exchange of the sums.
// A cluster's SMs are of one GPC, so 148 SMs hold 74 clusters of two CTAs but not 37 of four (33 on the B200 that was timed): the
// caller gives both numbers.  One cluster too many is a second wave: 100 rows x K 4096 in 33 / 34 tiles of 64 columns, cut in four
// 6.8 / 12.1, in two 8.0 / 8.0; of 128 columns 8.5 / 15.1 and 9.6 / 9.6; 74 tiles cut in two 8.5 and 10.5, whole 11.7 and 12.9.
// 128 columns whole / 2 / 4, then 64 columns whole / 2 / 4: 16 x 512 x 4096 12.1 / 9.5 / 8.0, 11.3 / 8.0 / 6.6; 100 x 4096 x 4096 13.1 / 10.2 /
// 8.8, 12.3 / 8.7 / -; 333 x 1792 x 4096 13.3 / 10.5 / -, 12.5 / - / -; 128 x 2048 x 2048 8.3 / 7.5 / 7.5, 7.7 / 6.3 / 6.0; but eight slices
// are in flight at once anyway: 16 x 512 x 1024 5.1 / 6.3 / 6.6, 4.7 / 5.2 / 5.3.
static int fp8Plan(int M, int N, int nK, int sms, int pairs, int quads, int *cutOut) {
  const int m1 = (M + 127) / 128, m2 = (M + 255) / 256;
  auto waves = [](long long tiles, int slots) { return (double)((tiles + slots - 1) / slots); };
  double best = waves((long long)m2 * ((N + 255) / 256), sms / 2) * (nK * 562.0 + 600);
  int tile = 0, cut = 1;
  for (int bn : {128, 64}) {
    const long long tiles = (long long)m1 * ((N + bn - 1) / bn);
    for (int c = 1; c <= (nK >= 12 ? 4 : 1); c *= 2) {
      const int per = (nK + c - 1) / c;
      if (c > 1 && (tiles > (c == 2 ? pairs : quads) || (c - 1) * per >= nK)) continue;
      const double w = waves(tiles * c, sms), slice = bn == 128 ? (w > 1 ? 320 : 283) : (w > 1 ? 260 : 246), turn = bn == 128 ? 800 : 600;
      const double exchange = c == 1 ? 0 : bn == 128 ? (c == 2 ? 1890 : 2700) : (c == 2 ? 660 : 1210);
      const double time = w * per * slice + (w - 1) * turn + exchange;
      if (time < best) {
        best = time;
        tile = bn;
        cut = c;
      }
    }
  }
  *cutOut = cut;
  return tile;
}
// The rule by itself: `pairs` clusters of two CTAs or `quads` of four are on the chip at once (0: not cut that way).
extern "C" int fcxGemmFp8PlanFor(int M, int N, int K, int sms, int pairs, int quads, int *cut) { return fp8Plan(M, N, K / 128, sms, pairs, quads, cut); }

namespace {

// How many clusters of `cut` CTAs the current device holds at once.  Both widths' kernels fill an SM, so one is asked for both.
// Without a device: eight GPCs of whole pairs of SMs, each of which may leave a pair over.
int clustersAtOnce(int cut) {
  static std::atomic<int> known[2][fcxhost::MAX_DEVICES];
  const int dev = fcxhost::currentDevice(), which = cut == 2 ? 0 : 1;
  int n = dev < fcxhost::MAX_DEVICES ? known[which][dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n - 1;
  const auto kernel = gemmFp8Kernel<128, true>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cut);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smemBytes(128);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cut;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  n = -1;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes(128)) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 0) {
    cudaGetLastError();
    return cut == 2 ? smCount() / 2 : std::max(0, smCount() - 16) / 4;
  }
  if (dev < fcxhost::MAX_DEVICES) known[which][dev].store(n + 1, std::memory_order_relaxed);
  return n;
}

}  // namespace

// The plan of a launch on the current device.
extern "C" int fcxGemmFp8Plan(int M, int N, int K, int sms, int *cut) {
  return fcxGemmFp8PlanFor(M, N, K, sms, std::min(clustersAtOnce(2), sms / 2), std::min(clustersAtOnce(4), sms / 4), cut);
}
// The tile of a long sum that is not cut, as the tables of timings above have it; launches ask fcxGemmFp8Plan.
extern "C" int fcxGemmFp8Tile(int M, int N, int sms) {
  int cut;
  return fp8Plan(M, N, 32, sms, 0, 0, &cut);
}

extern "C" cudaError_t fcxGemmFp8Blockwise(const void *aq, const float *sa, const void *bq, const float *sb, void *c, int M, int N, int K,
                                           int ldc, int *errFlag, cudaStream_t s) {
  if (K % 128 || ldc % 8 || M <= 0 || N <= 0 || K <= 0) return cudaErrorInvalidValue;
  if (((uintptr_t)aq | (uintptr_t)bq | (uintptr_t)c) & 15) return cudaErrorInvalidValue;
  CUtensorMap ma, mc;
  if (!makeTileMap(&ma, aq, M, K, K, BM, 1) || !makeStoreMap(&mc, c, M, N, ldc)) return cudaErrorNotSupported;
  Params p{};
  p.M = M; p.N = N; p.K = K; p.sa = sa; p.sb = sb; p.errFlag = errFlag;
  int cut = 1;
  const int tile = fcxGemmFp8Plan(M, N, K, smCount(), &cut);
  p.group = tile == 0 ? 8 : (N + 127) / 128 >= 48 ? 16 : 8;
  if (tile == 0) return launchPair(ma, bq, mc, p, s);
  if (tile == 128) return cut > 1 ? launchOne<128, true>(ma, bq, mc, p, cut, s) : launchOne<128, false>(ma, bq, mc, p, 1, s);
  return cut > 1 ? launchOne<64, true>(ma, bq, mc, p, cut, s) : launchOne<64, false>(ma, bq, mc, p, 1, s);
}

extern "C" cudaError_t fcxQuantFp8Act(const void *x, void *q, float *sa, int M, int K, int ldx, cudaStream_t s) {
  if (K % 128 || ldx % 4) return cudaErrorInvalidValue;
  const size_t blocks = (size_t)M * (K / 128);
  if (blocks == 0) return cudaSuccess;
  const bool wide = ldx % 8 == 0 && ((uintptr_t)x & 15) == 0;
  const __nv_bfloat16 *src = (const __nv_bfloat16 *)x;
  __nv_fp8_storage_t *dst = (__nv_fp8_storage_t *)q;
  // four blocks per lane group once that still leaves two CTAs for every SM, else one: a small batch wants many CTAs
  if (wide && blocks >= 16 * 4 * 2 * (size_t)smCount()) return fcxpdl::launchPdl(quantActKernel<8, 4>, (unsigned)((blocks + 63) / 64), 256, 0, s, src, dst, sa, M, K, ldx);
  if (wide) return fcxpdl::launchPdl(quantActKernel<8, 1>, (unsigned)((blocks + 15) / 16), 256, 0, s, src, dst, sa, M, K, ldx);
  return fcxpdl::launchPdl(quantActKernel<4, 1>, (unsigned)((blocks + 7) / 8), 256, 0, s, src, dst, sa, M, K, ldx);
}

extern "C" cudaError_t fcxQuantFp8Weight(const void *w, void *q, float *sb, int N, int K, int ldw, cudaStream_t s) {
  if (K % 128 || ldw % 4) return cudaErrorInvalidValue;
  quantWeightKernel<<<((N + 127) / 128) * (K / 128), 256, 0, s>>>((const __nv_bfloat16 *)w, (__nv_fp8_storage_t *)q, sb, N, K, ldw);
  return cudaGetLastError();
}

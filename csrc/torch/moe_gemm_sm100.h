// Launchers of the expert MLP's grouped GEMMs (moe_gemm_sm100.cu): all local experts in one launch.
#pragma once
#include "../kernels/devcomm.h"
#include <cuda_runtime_api.h>
#include <stdint.h>

#define FCX_MOE_MAX_EXPERTS 64  // experts of the whole job, and so the most that one rank can hold

#ifdef __cplusplus
extern "C" {
#endif
// h[r, :] = silu(x[r] wg^T) * (x[r] wu^T) for the first rows[l] rows of each of the L segments of capL rows.
// x [L * capL, H] and h [L * capL, F] bf16, contiguous; w: L matrices [2F, H] (gate rows, then up rows), `ldw` elements
// between rows.  Rows of a segment past rows[l] may be overwritten in h up to the next multiple of 32.
cudaError_t fcxMoeUpGrouped(const void *x, const void *const *w, void *h, const int *rows, int L, int capL, int H, int F, const int *ldw,
                            int *errFlag, cudaStream_t s);
// y = h[r] w^T (h bf16, `ldh` elements between rows), stored at its token's place on the rank it came from: heap[info[r].x] + combineOff + (info[r].y * topk + info[r].z)
// * H elements.  w: L matrices [H, F].  Afterwards every CTA of the launch (gridOut of them) adds 1 to the u64 counter at
// doneOff on every rank.
cudaError_t fcxMoeDownGrouped(const FcxDevComm *dc, const void *h, const void *const *w, const int *rows, int L, int capL, int H, int F, int ldh,
                              const int *ldw, const void *rowInfo, size_t combineOff, size_t doneOff, int topk, int *errFlag, int *gridOut,
                              cudaStream_t s);
// Accumulator columns of a tile (256 or 128) for that many 256-row blocks and columns and sums of length K; the kernels decide for
// themselves.
int fcxMoeTileColumns(int rowBlocks, int cols, int K, int up, int pairs);
#ifdef __cplusplus
}
#endif

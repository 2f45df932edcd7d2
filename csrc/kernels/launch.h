// Host-callable launchers of the collective kernels (implemented in
// collectives.cu) and launch-shape constants shared with the runtime.
#pragma once
#include "devcomm.h"
#include <cuda_runtime_api.h>

#define FCX_THREADS 512

// What an emulated collective needs to know of every rank; a kernel argument (no copy to the device before the launch).
struct FcxEmuRanks {
  FcxDevComm dc[FCX_MAX_RANKS];
  FcxCollArgs args[FCX_MAX_RANKS];
};

#ifdef __cplusplus
extern "C" {
#endif
cudaError_t fcxLaunchColl(const FcxDevComm *dc, const FcxCollArgs *a, int nctas, cudaStream_t s);
// zero-copy kinds (zerocopy.cu); fcxLaunchColl forwards to these
cudaError_t fcxLaunchZc(const FcxDevComm *dc, const FcxCollArgs *a, int nctas, cudaStream_t s);
cudaError_t fcxLaunchZcEmu(const FcxEmuRanks *l, int nranks, int nctas, cudaStream_t s);
// low-latency reductions (lowlatency.cu); fcxLaunchColl forwards to these, too
cudaError_t fcxLaunchLl(const FcxDevComm *dc, const FcxCollArgs *a, int nctas, cudaStream_t s);
cudaError_t fcxLaunchLlEmu(const FcxEmuRanks *l, int nranks, int nctas, cudaStream_t s);
cudaError_t fcxLaunchP2p(const FcxDevComm *dc, const FcxP2pArgs *g, cudaStream_t s);
cudaError_t fcxLaunchWaitTest(const FcxDevComm *dc, uint64_t want, cudaStream_t s);
// Single-GPU emulation of `nranks` ranks in one cooperative launch.  The ranks' descriptors and arguments travel in the
// launch itself; dcs and gs are device arrays with one entry per emulated rank.
cudaError_t fcxLaunchCollEmu(const FcxEmuRanks *l, int nranks, int nctas, cudaStream_t s);
cudaError_t fcxLaunchP2pEmu(const FcxDevComm *dcs, const FcxP2pArgs *gs, int nranks, int ctasPerRank, cudaStream_t s);
#ifdef __cplusplus
}
#endif

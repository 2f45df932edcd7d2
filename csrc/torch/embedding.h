// Launchers of the token + position embedding (embedding.cu).  bf16 tables, int64 tokens.
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

constexpr int EMB_MAX_TOKENS = 16384;

#ifdef __cplusplus
extern "C" {
#endif
int fcxEmbeddingTakes(int64_t M, int64_t C);
// x[i] = wte[tokens[i]] + wpe[i % T] for M rows of C columns; V rows of wte
cudaError_t fcxEmbeddingFwd(const int64_t *tokens, const void *wte, const void *wpe, void *x, int M, int T, int C, int V, cudaStream_t s);
// adds the gradients to dwte [V, C] and dwpe [T or more, C]; either may be null
cudaError_t fcxEmbeddingBwd(const void *dx, const int64_t *tokens, void *dwte, void *dwpe, int M, int T, int C, int V, cudaStream_t s);
#ifdef __cplusplus
}
#endif

// Launch interface of the tcgen05 small-M GEMM (kTcMinTokens or more token rows).
#pragma once

#include "gemv.cuh"
#include "mma_common.cuh"

namespace gufo {

// Fewest token rows that take this path: a third pass over the weights on the
// eight-token GEMV kernels. Those keep the activations to 24 bits and this path
// rounds them to fp16, so the line stays where it is although two passes are
// slower than this.
constexpr int kTcMinTokens = 17;

// Whether a product of `tokens` rows against parts of `type` runs on this path.
bool TcGemmRuns(const gufo_cuda_ctx* ctx, int type, int cols, int tokens);

// Enqueues y = [W_0 x | W_1 x | ...] for `tokens` >= kTcMinTokens rows; every
// part of `base` must satisfy TcGemmRuns. x is 16-byte aligned.
int LaunchGemmTc(gufo_cuda_ctx* ctx, const GemvArgs& base, int tokens);

// Reads (after synchronizing the stream) the code a bounded wait of the GEMM
// kernel left when it ran out; 0 when none did.
int TcGemmError(gufo_cuda_ctx* ctx, int* code);

}  // namespace gufo

// The one-launch quantizers of short calls (quantize_call.cu) as the other host files see them.
#pragma once

#include "capi.h"

namespace unica {

// Up to this many tokens a cluster of eight blocks takes a head's statistics and quantizes it in one launch: the tokens come
// out of L2 the second time, and eight blocks are enough to read a head of 2 MB in a few microseconds.  Above it the persistent
// kernels of quantize_fused.cu, or the separate passes, keep more of the GPU on a head.
constexpr int CALL_TOKENS = 8192;

// One operand of a call; x null: the call does not quantize it.
struct CallOperand {
    const __nv_bfloat16* x;
    TokenLayout in;
    int n_tokens, tiles;
    uint8_t* codes;
    void* scales;  // INT8: float per tile (Q, K) or channel (V); NVFP4: the scale bytes
    float* mean;   // K: [heads][128]; NVFP4 Q: [heads][groups][128]
    float* outer;  // NVFP4: per head (Q, K) or channel (V)
};
struct CallQuantize {
    CallOperand q, k, v;
    RopeTable rope;  // Q and K
    int heads;
    int v_mode;          // INT8: UNICA_B200_V_*
    float* v_token;      // per token
    int n_outliers;      // outliers
    int* outlier_keys;   // [heads][n_outliers]
    float* outlier_rows;  // [heads][n_outliers][128]
    int smooth;          // NVFP4: tokens per group of Q's means, a multiple of 256
};
// launches: counts them, or null
int quantize_call_int8(const CallQuantize& call, cudaStream_t stream, int* launches = nullptr);
int quantize_call_fp4(const CallQuantize& call, cudaStream_t stream);

}  // namespace unica

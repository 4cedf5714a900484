// Host-side plumbing shared by the C entry points: the thread-local error message and launch checks.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/unica_b200.h"
#include "common.cuh"

int unica_fail(int code, const char* message);
int unica_check_launch(const char* what);  // cudaGetLastError after a launch -> 0 or UNICA_B200_ERR_CUDA
int unica_check_device();                  // the current device must be compute capability 10.0 (cached per device)
int unica_sm_count(int* sms);              // of the current device (cached per device)

// Launches a kernel that begins with wait_for_previous_kernel(), overlapped with the end of the one before it in the stream
// (one of this library's that starts only when ITS predecessor is complete, or waits for it, before it lets this one in; or, where the
// kernel lets nobody in before its wait, any).
template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool overlapped, Args&&... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid, config.blockDim = dim3(threads), config.dynamicSmemBytes = smem, config.stream = stream;
    cudaLaunchAttribute overlap = {};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &overlap, config.numAttrs = overlapped ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Args&&>(args)...);
}

// The attention kernels behind their entry points.  k_outer: null, or the per-head factor that qk_outer still lacks.
// overlapped: the launch before is the call's own (see launch_after).
int unica_attention_int8(const int8_t* q8, const float* q_scale, const int8_t* k8, const float* k_scale, const int8_t* v8, const float* v_scale,
                         const float* v_token, int v_mode, const int* outlier_keys, const float* outlier_rows, int n_outliers, void* out,
                         void* const* peer_out, int n_peers, unica_token_layout out_layout, int heads, int n_queries, int n_keys, float scale_log2,
                         int* status, void* stream, bool overlapped = false);
int unica_attention_fp4(const uint8_t* q4, const void* sfq, const uint8_t* k4, const void* sfk, const uint8_t* v4, const void* sfv,
                        const float* qk_outer, const float* k_outer, const float* v_outer, const float* bias, int q_blocks, int smooth_q, void* out,
                        void* const* peer_out, int n_peers, unica_token_layout out_layout, int heads, int n_queries, int n_keys, float scale_log2,
                        uint32_t* p_words, int* status, void* stream, bool overlapped = false);

// The smoothing table behind its entry points; rope: null or the table.
int unica_smooth_bias(const void* k, unica_token_layout layout, const float* k_mean, const float* q_mean, unica::RopeTable rope, int heads, int q_blocks,
                      int n_keys, float scale_log2, float* bias, int* status, void* stream, bool overlapped = false);

// Checks and copies a caller's list of peer output tensors (see PeerOutputs); n_peers == 0 leaves `peers` empty.
static inline int unica_peer_outputs(const void* out, void* const* peer_out, int n_peers, unica::PeerOutputs* peers) {
    peers->count = 0;
    if (n_peers == 0) return UNICA_B200_OK;
    if (n_peers < 0 || n_peers > unica::MAX_PEER_OUTPUTS || !peer_out) return unica_fail(UNICA_B200_ERR_ARGUMENT, "peer outputs: n_peers must be in 0..7 with a pointer list");
    for (int i = 0; i < n_peers; ++i) {
        if (!peer_out[i] || reinterpret_cast<uintptr_t>(peer_out[i]) % 16 || peer_out[i] == out)
            return unica_fail(UNICA_B200_ERR_ARGUMENT, "peer outputs: every pointer must be non-null, 16-byte aligned and different from out");
        peers->out[i] = static_cast<__nv_bfloat16*>(peer_out[i]);
    }
    peers->count = n_peers;
    return UNICA_B200_OK;
}

static inline unica::TokenLayout to_layout(const unica_token_layout& l) {
    unica::TokenLayout t;
    t.batch = l.batch, t.head = l.head, t.token = l.token, t.heads = l.heads, t.half = l.dtype == UNICA_B200_FLOAT16;
    return t;
}

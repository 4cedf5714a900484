// A whole call of attention() behind one entry point: operands in a workspace of the caller's, every launch from here.
//
// Through the entry points of the single steps a call costs its Python caller a dozen small allocations and as many trips
// through ctypes, some 100 us of host time: more than the GPU needs for 4 heads x 1024 tokens.
#include <algorithm>

#include "quantize_call.h"

using namespace unica;

namespace {

// What a call keeps in its workspace, 256-byte aligned; base 0: only the size is wanted.
struct Plan {
    size_t used = 0;
    uint8_t* base = nullptr;
    template <typename T>
    T* take(long long count) {
        T* at = reinterpret_cast<T*>(base + used);
        used = (used + size_t(count) * sizeof(T) + 255) & ~size_t(255);
        return at;
    }
    int q_tiles, k_tiles, groups;  // groups of Q's means
    bool short_q, short_k;         // the one-launch quantizer takes Q / K and V
    // INT8
    int8_t *q8, *k8, *v8;
    float *q_scale, *k_scale, *k_mean, *v_scale, *v_token, *outlier_rows;
    int* outlier_keys;
    // NVFP4
    uint8_t *q4, *q_sf, *k4, *k_sf, *v4, *v_sf;
    float *q_outer, *k_outer, *v_outer, *q_mean, *bias;
    // scratch of the separate passes
    void* fused;
    float *partial, *stats;  // partial sums; low and high (and unwanted means) of one tensor

    Plan(const unica_b200_call& c, void* workspace) : base(static_cast<uint8_t*>(workspace)) {
        const long long heads = c.heads, stats_blocks = (std::max(c.n_queries, c.n_keys) + 255) / 256;
        q_tiles = (c.n_queries + 2 * QUERY_TILE - 1) / (2 * QUERY_TILE) * 2;
        k_tiles = (c.n_keys + KEY_TILE - 1) / KEY_TILE;
        groups = c.smooth_q > 0 ? (c.n_queries + c.smooth_q - 1) / c.smooth_q : 1;
        short_q = c.n_queries <= CALL_TOKENS, short_k = c.n_keys <= CALL_TOKENS;
        if (c.kernel == UNICA_B200_FAST) {
            short_q = short_k = short_q && short_k && c.smooth_q > 0;  // all or nothing
            q4 = take<uint8_t>(heads * q_tiles * QUERY_TILE * HEAD_DIM / 2), q_sf = take<uint8_t>(heads * q_tiles * QUERY_TILE * 8);
            k4 = take<uint8_t>(heads * k_tiles * KEY_TILE * HEAD_DIM / 2), k_sf = take<uint8_t>(heads * k_tiles * KEY_TILE * 8);
            v4 = take<uint8_t>(heads * k_tiles * 144 * 32), v_sf = take<uint8_t>(heads * k_tiles * 1024);
            q_outer = take<float>(heads), k_outer = take<float>(heads), v_outer = take<float>(heads * HEAD_DIM);
            k_mean = take<float>(heads * HEAD_DIM), q_mean = take<float>(heads * groups * HEAD_DIM);
            bias = c.smooth_q > 0 ? take<float>(heads * groups * k_tiles * KEY_TILE) : nullptr;
            if (!short_k) partial = take<float>(heads * stats_blocks * 3 * HEAD_DIM), stats = take<float>(heads * groups * 3 * HEAD_DIM);
        } else {
            q8 = take<int8_t>(heads * q_tiles * QUERY_TILE * HEAD_DIM), q_scale = take<float>(heads * q_tiles);
            k8 = take<int8_t>(heads * k_tiles * KEY_TILE * HEAD_DIM), k_scale = take<float>(heads * k_tiles), k_mean = take<float>(heads * HEAD_DIM);
            v8 = take<int8_t>(heads * k_tiles * KEY_TILE * HEAD_DIM), v_scale = take<float>(heads * HEAD_DIM);
            v_token = c.v_mode == UNICA_B200_V_TOKEN ? take<float>(heads * k_tiles * 2 * KEY_TILE) : nullptr;
            outlier_keys = nullptr, outlier_rows = nullptr;
            if (c.v_mode == UNICA_B200_V_OUTLIERS) outlier_keys = take<int>(heads * c.n_outliers), outlier_rows = take<float>(heads * c.n_outliers * HEAD_DIM);
            if (!short_k) {
                fused = take<uint8_t>(UNICA_B200_FUSED_SCRATCH_BYTES);
                if (c.rope) partial = take<float>(heads * stats_blocks * 3 * HEAD_DIM), stats = take<float>(heads * 3 * HEAD_DIM);
            }
        }
    }
};

CallOperand operand(const void* x, const unica_token_layout& layout, int n_tokens, int tiles, void* codes, void* scales, float* mean, float* outer) {
    return CallOperand{static_cast<const __nv_bfloat16*>(x), to_layout(layout), n_tokens, tiles, static_cast<uint8_t*>(codes), scales, mean, outer};
}

int check(const unica_b200_call* c) {
    if (!c) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: null pointer");
    if (c->heads <= 0 || c->heads > 65535 || c->n_queries <= 0 || c->n_keys <= 0)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: heads must be in 1..65535, n_queries and n_keys positive");
    if (c->kernel != UNICA_B200_ACCURATE && c->kernel != UNICA_B200_FAST) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: unknown kernel");
    if (c->kernel == UNICA_B200_FAST && (c->smooth_q < 0 || c->smooth_q % 256))
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: smooth_q must be 0 or a multiple of 256");
    if (c->kernel == UNICA_B200_ACCURATE && c->v_mode == UNICA_B200_V_OUTLIERS && (c->n_outliers < 1 || c->n_outliers > 8 || c->n_keys > CALL_TOKENS))
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: 1..8 outliers, and at most 8192 keys (the outlier keys of longer calls are the caller's to find)");
    return UNICA_B200_OK;
}

int call_accurate(const unica_b200_call& c, const Plan& p, int* launches) {
    const RopeTable rope{static_cast<const __half*>(c.rope), c.rope_batch_stride};
    CallQuantize quantize = {};
    quantize.rope = rope, quantize.heads = c.heads, quantize.v_mode = c.v_mode, quantize.v_token = p.v_token;
    quantize.n_outliers = c.n_outliers, quantize.outlier_keys = p.outlier_keys, quantize.outlier_rows = p.outlier_rows;
    if (p.short_q) quantize.q = operand(c.q, c.q_layout, c.n_queries, p.q_tiles, p.q8, p.q_scale, nullptr, nullptr);
    if (p.short_k) {
        quantize.k = operand(c.k, c.k_layout, c.n_keys, p.k_tiles, p.k8, p.k_scale, p.k_mean, nullptr);
        quantize.v = operand(c.v, c.v_layout, c.n_keys, p.k_tiles, p.v8, p.v_scale, nullptr, nullptr);
    }
    if (p.short_q || p.short_k) {
        if (int e = quantize_call_int8(quantize, static_cast<cudaStream_t>(c.stream), launches)) return e;
    }
    if (!p.short_q) {
        if (int e = c.rope ? unica_b200_quantize_int8_rope(c.q, c.q_layout, nullptr, c.rope, c.rope_batch_stride, c.heads, c.n_queries, QUERY_TILE, p.q_tiles, p.q8,
                                                           p.q_scale, c.stream)
                           : unica_b200_quantize_q_int8_stream(c.q, c.q_layout, c.heads, c.n_queries, p.q_tiles, p.q8, p.q_scale, c.stream))
            return e;
        ++*launches;
    }
    if (!p.short_k) {
        if (c.rope) {
            float* spare = p.stats + size_t(c.heads) * HEAD_DIM;
            if (int e = unica_b200_channel_stats_rope(c.k, c.k_layout, c.rope, c.rope_batch_stride, c.heads, c.n_keys, 0, p.partial, p.k_mean, p.stats, spare, c.stream))
                return e;
            if (int e = unica_b200_quantize_int8_rope(c.k, c.k_layout, p.k_mean, c.rope, c.rope_batch_stride, c.heads, c.n_keys, KEY_TILE, p.k_tiles, p.k8, p.k_scale,
                                                      c.stream))
                return e;
            *launches += 3;
        } else {
            if (int e = unica_b200_quantize_k_int8_fused(c.k, c.k_layout, c.heads, c.n_keys, p.k_tiles, p.fused, UNICA_B200_FUSED_SCRATCH_BYTES, p.k8, p.k_scale,
                                                         p.k_mean, c.status, c.stream))
                return e;
            ++*launches;
        }
        if (int e = c.v_mode == UNICA_B200_V_TOKEN
                        ? unica_b200_quantize_v_int8(c.v, c.v_layout, nullptr, nullptr, nullptr, 1, c.heads, c.n_keys, p.v8, p.v_scale, p.v_token, c.stream)
                        : unica_b200_quantize_v_int8_fused(c.v, c.v_layout, c.heads, c.n_keys, p.fused, UNICA_B200_FUSED_SCRATCH_BYTES, p.v8, p.v_scale, c.status, c.stream))
            return e;
        ++*launches;
    }
    ++*launches;
    return unica_attention_int8(p.q8, p.q_scale, p.k8, p.k_scale, p.v8, p.v_scale, p.v_token, c.v_mode, p.outlier_keys, p.outlier_rows, c.n_outliers, c.out, c.peer_out,
                                c.n_peers, c.out_layout, c.heads, c.n_queries, c.n_keys, c.scale_log2, c.status, c.stream, true);
}

int call_fast(const unica_b200_call& c, const Plan& p, int* launches) {
    const RopeTable rope{static_cast<const __half*>(c.rope), c.rope_batch_stride};
    if (p.short_k) {
        CallQuantize quantize = {};
        quantize.rope = rope, quantize.heads = c.heads, quantize.smooth = c.smooth_q;
        quantize.q = operand(c.q, c.q_layout, c.n_queries, p.q_tiles, p.q4, p.q_sf, p.q_mean, p.q_outer);
        quantize.k = operand(c.k, c.k_layout, c.n_keys, p.k_tiles, p.k4, p.k_sf, p.k_mean, p.k_outer);
        quantize.v = operand(c.v, c.v_layout, c.n_keys, p.k_tiles, p.v4, p.v_sf, nullptr, p.v_outer);
        if (int e = quantize_call_fp4(quantize, static_cast<cudaStream_t>(c.stream))) return e;
        ++*launches;
    } else {
        auto stats = [&](const void* x, const unica_token_layout& layout, bool rotated, int n, int per, int n_groups, float* mean, float** low, float** high) -> int {
            float* spare = p.stats;
            *low = spare + size_t(c.heads) * n_groups * HEAD_DIM, *high = *low + size_t(c.heads) * n_groups * HEAD_DIM;
            *launches += 2;
            return rotated && c.rope ? unica_b200_channel_stats_rope(x, layout, c.rope, c.rope_batch_stride, c.heads, n, per, p.partial, mean ? mean : spare, *low, *high, c.stream)
                                     : unica_b200_channel_stats(x, layout, c.heads, n, per, p.partial, mean ? mean : spare, *low, *high, c.stream);
        };
        auto rows = [&](const void* x, const unica_token_layout& layout, const float* mean, int mean_tokens, const float* outer, int n, int per_tile, int tiles, uint8_t* codes,
                        uint8_t* sf) -> int {
            ++*launches;
            return c.rope ? unica_b200_quantize_fp4_rows_rope(x, layout, mean, mean_tokens, c.rope, c.rope_batch_stride, outer, c.heads, n, per_tile, tiles, codes, sf, c.stream)
                          : unica_b200_quantize_fp4_rows(x, layout, mean, mean_tokens, outer, c.heads, n, per_tile, tiles, codes, sf, c.stream);
        };
        float *low, *high;
        const float* q_mean = c.smooth_q > 0 ? p.q_mean : nullptr;
        if (int e = stats(c.k, c.k_layout, true, c.n_keys, 0, 1, p.k_mean, &low, &high)) return e;
        if (int e = unica_b200_nvfp4_outer(p.k_mean, low, high, c.heads, 1, p.k_outer, c.stream)) return e;
        if (int e = rows(c.k, c.k_layout, p.k_mean, 0, p.k_outer, c.n_keys, KEY_TILE, p.k_tiles, p.k4, p.k_sf)) return e;
        if (int e = stats(c.q, c.q_layout, true, c.n_queries, c.smooth_q, p.groups, p.q_mean, &low, &high)) return e;
        if (int e = unica_b200_nvfp4_outer(q_mean, low, high, c.heads, p.groups, p.q_outer, c.stream)) return e;
        if (int e = rows(c.q, c.q_layout, q_mean, c.smooth_q, p.q_outer, c.n_queries, QUERY_TILE, p.q_tiles, p.q4, p.q_sf)) return e;
        if (int e = stats(c.v, c.v_layout, false, c.n_keys, 0, 1, nullptr, &low, &high)) return e;
        if (int e = unica_b200_quantize_v_fp4(c.v, c.v_layout, low, high, c.heads, c.n_keys, p.v4, p.v_sf, p.v_outer, c.stream)) return e;
        *launches += 3;
    }
    if (p.bias) {
        if (int e = unica_smooth_bias(c.k, c.k_layout, p.k_mean, p.q_mean, rope, c.heads, p.groups, c.n_keys, c.scale_log2, p.bias, c.status, c.stream, true)) return e;
        ++*launches;
    }
    ++*launches;
    return unica_attention_fp4(p.q4, p.q_sf, p.k4, p.k_sf, p.v4, p.v_sf, p.q_outer, p.k_outer, p.v_outer, p.bias, p.bias ? p.groups : 0, c.smooth_q, c.out, c.peer_out, c.n_peers,
                               c.out_layout, c.heads, c.n_queries, c.n_keys, c.scale_log2, nullptr, c.status, c.stream, true);
}

}  // namespace

extern "C" int unica_b200_attention_workspace(const unica_b200_call* call, size_t* bytes) {
    if (int e = check(call)) return e;
    if (!bytes) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_workspace: null pointer");
    *bytes = Plan(*call, nullptr).used;
    return UNICA_B200_OK;
}

extern "C" int unica_b200_attention_call(const unica_b200_call* call, int* launches) {
    if (int e = check(call)) return e;
    if (!call->q || !call->k || !call->v || !call->out || !call->workspace || !call->status || !launches)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: null pointer");
    const Plan plan(*call, call->workspace);
    if (plan.used > call->workspace_bytes || reinterpret_cast<uintptr_t>(call->workspace) % 256)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_call: the workspace must be 256-byte aligned and hold unica_b200_attention_workspace() bytes");
    *launches = 0;
    return call->kernel == UNICA_B200_FAST ? call_fast(*call, plan, launches) : call_accurate(*call, plan, launches);
}

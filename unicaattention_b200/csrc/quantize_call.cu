// The quantization of a short call (up to CALL_TOKENS tokens) in ONE launch: Q, K and V of all heads, statistics included.
//
// The separate passes need three to eight launches for this, each a few microseconds on the device and as many on the host:
// for 4 heads x 1024 tokens that was most of the call.  Here the grid is made of clusters of eight blocks, each of which is
// given a head's K, a head's V or (NVFP4) a head's Q, and in INT8 eight tiles of Q, which need no statistics:
//   1. the blocks of a cluster take the statistics of an eighth of the head's 256-token blocks each,
//   2. they read one another's partial results through distributed shared memory, all in the same order,
//   3. and quantize an eighth of the head's tiles each; the tokens come out of L2 now.
// What bounds it: latency (two dependent trips to memory and a cluster barrier each way).
//
// Sums run in the order of channel_stats_kernel and its finish kernel (quantize.cu), minima and maxima are exact: the
// operands are bit for bit those of the separate passes.
#include <cooperative_groups.h>

#include <type_traits>

#include "quantize_call.h"
#include "quantize_fp4.cuh"
#include "quantize_int8.cuh"

namespace unica {

namespace cg = cooperative_groups;

constexpr int CALL_CLUSTER = 8, CALL_THREADS = 256;
constexpr int CALL_LANES = 16, CALL_BLOCK = 256;  // statistics: 16 token lanes, 256 tokens per partial sum, as in quantize.cu
constexpr int CALL_PARTS = CALL_TOKENS / CALL_BLOCK / CALL_CLUSTER;  // partial sums per block at most
constexpr int CALL_OUTLIERS = 8;
constexpr int CALL_GROUPS = CALL_PARTS + 2;  // groups of Q's means that a block's eighth of the tiles can touch
static_assert(CALL_THREADS == THREADS && CALL_THREADS == FP4_THREADS && CALL_THREADS == CALL_LANES * (HEAD_DIM / 8), "one block shape for all tile routines");

struct CallStats {
    float part[CALL_PARTS][3][HEAD_DIM];  // sum, min, max of this block's 256-token blocks
    union {  // one after the other
        float lanes[3][CALL_LANES][HEAD_DIM];                              // the token lanes' sums on their way to one
        VTileSmem v_tile;                                                  // a tile of V on its way round
        unsigned long long candidates[CALL_TOKENS / CALL_CLUSTER + 1];  // the block's tokens, see find_outliers
    };
    float mean[HEAD_DIM], low[HEAD_DIM], high[HEAD_DIM];
    float scratch[CALL_THREADS / 32];
};
// this block's share of `count` things
__device__ __forceinline__ int share(int count, int rank) { return count * rank / CALL_CLUSTER; }

// Sum, min and max per channel of 256-token block `b` into part[3][128]: channel_stats_kernel's arithmetic.
template <typename Skip>
__device__ __forceinline__ void block_stats(const __nv_bfloat16* __restrict__ x, const TokenLayout& in, const RopeTable& rope, Skip skip, int head, int b,
                                            int n_tokens, CallStats& sm, float (&part)[3][HEAD_DIM]) {
    const int chunk = threadIdx.x % 16, lane = threadIdx.x / 16;
    float sum[8], low[8], high[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) sum[i] = 0.0f, low[i] = INFINITY, high[i] = -INFINITY;
    const int end = min((b + 1) * CALL_BLOCK, n_tokens);
#pragma unroll 8
    for (int token = b * CALL_BLOCK + lane; token < end; token += CALL_LANES) {
        float v[8];
        load8(v, x + in.offset(head, token) + chunk * 8, in.half);
        if (skip(token)) continue;
        if (rope.table) rope8(v, rope.row(in, head, token), chunk * 8);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            sum[i] += v[i];
            low[i] = fminf(low[i], v[i]);
            high[i] = fmaxf(high[i], v[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        sm.lanes[0][lane][chunk * 8 + i] = sum[i];
        sm.lanes[1][lane][chunk * 8 + i] = low[i];
        sm.lanes[2][lane][chunk * 8 + i] = high[i];
    }
    __syncthreads();
    if (threadIdx.x < HEAD_DIM) {
        float s = 0.0f, lo = INFINITY, hi = -INFINITY;
        for (int l = 0; l < CALL_LANES; ++l) {
            s += sm.lanes[0][l][threadIdx.x];
            lo = fminf(lo, sm.lanes[1][l][threadIdx.x]);
            hi = fmaxf(hi, sm.lanes[2][l][threadIdx.x]);
        }
        part[0][threadIdx.x] = s, part[1][threadIdx.x] = lo, part[2][threadIdx.x] = hi;
    }
    __syncthreads();
}

// The head's mean, min and max into sm of every block of the cluster.  Every thread of the cluster calls it.
template <typename Skip>
__device__ __forceinline__ void head_stats(const __nv_bfloat16* __restrict__ x, const TokenLayout& in, const RopeTable& rope, Skip skip, int head,
                                           int n_tokens, int rank, CallStats& sm) {
    const int blocks = (n_tokens + CALL_BLOCK - 1) / CALL_BLOCK, b0 = share(blocks, rank), b1 = share(blocks, rank + 1);
    for (int b = b0; b < b1; ++b) block_stats(x, in, rope, skip, head, b, n_tokens, sm, sm.part[b - b0]);
    cg::this_cluster().sync();
    if (threadIdx.x < HEAD_DIM) {
        float s = 0.0f, lo = INFINITY, hi = -INFINITY;
        for (int r = 0; r < CALL_CLUSTER; ++r) {
            const CallStats* theirs = cg::this_cluster().map_shared_rank(&sm, r);
            const int parts = share(blocks, r + 1) - share(blocks, r);
            for (int i = 0; i < parts; ++i) {
                s += theirs->part[i][0][threadIdx.x];
                lo = fminf(lo, theirs->part[i][1][threadIdx.x]);
                hi = fmaxf(hi, theirs->part[i][2][threadIdx.x]);
            }
        }
        sm.mean[threadIdx.x] = s / float(n_tokens), sm.low[threadIdx.x] = lo, sm.high[threadIdx.x] = hi;
    }
    __syncthreads();
}

// The n_outliers keys with the largest max |v| of the head, ties to the lower key (what the reference's emulation takes), in
// every block of the cluster: -1 where the head has fewer keys.
struct CallOutliers {
    unsigned long long mine[CALL_OUTLIERS];  // this block's candidates: max |v| as bits, then the complement of the key
    int keys[CALL_OUTLIERS];
};
__device__ __forceinline__ unsigned long long larger(unsigned long long a, unsigned long long b) { return a > b ? a : b; }
__device__ __forceinline__ unsigned long long warp_largest(unsigned long long x) {
#pragma unroll
    for (int d = 16; d > 0; d /= 2) x = larger(x, __shfl_xor_sync(0xffffffffu, x, d));
    return x;
}
__device__ __forceinline__ void find_outliers(const __nv_bfloat16* __restrict__ v, const TokenLayout& in, int head, int n_tokens, int n_outliers, int rank,
                                              unsigned long long* candidates, CallOutliers& sm) {
    const int t0 = share(n_tokens, rank), count = share(n_tokens, rank + 1) - t0;
    const int chunk = threadIdx.x % 16, lane = threadIdx.x / 16;
#pragma unroll 4
    for (int i = lane; i < (count + CALL_LANES - 1) / CALL_LANES * CALL_LANES; i += CALL_LANES) {
        float amax = 0.0f;
        if (i < count) {
            float x[8];
            load8(x, v + in.offset(head, t0 + i) + chunk * 8, in.half);
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(x[j]));
        }
#pragma unroll
        for (int d = 8; d > 0; d /= 2) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
        if (chunk == 0 && i < count) candidates[i] = (static_cast<unsigned long long>(__float_as_uint(amax)) << 32) | (0xffffffffu - unsigned(t0 + i));
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // one warp: the largest, n_outliers times
        for (int o = 0; o < n_outliers; ++o) {
            unsigned long long best = 0;
            for (int i = threadIdx.x; i < count; i += 32) best = larger(best, candidates[i]);
            best = warp_largest(best);
            if (threadIdx.x == 0) sm.mine[o] = best;
            for (int i = threadIdx.x; i < count; i += 32)
                if (candidates[i] == best) candidates[i] = 0;
            __syncwarp();
        }
    }
    cg::this_cluster().sync();
    if (threadIdx.x < 32) {
        unsigned long long mine[2];  // eight blocks' eight candidates, two per lane
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int i = threadIdx.x * 2 + j;
            mine[j] = i % CALL_OUTLIERS < n_outliers ? cg::this_cluster().map_shared_rank(&sm, i / CALL_OUTLIERS)->mine[i % CALL_OUTLIERS] : 0;
        }
        for (int o = 0; o < n_outliers; ++o) {
            const unsigned long long best = warp_largest(larger(mine[0], mine[1]));
            if (threadIdx.x == 0) sm.keys[o] = best ? int(0xffffffffu - unsigned(best)) : -1;
            if (mine[0] == best) mine[0] = 0;
            if (mine[1] == best) mine[1] = 0;
        }
    }
    __syncthreads();
}

struct NoSkip {
    __device__ __forceinline__ bool operator()(int) const { return false; }
};
struct SkipKeys {
    const int* keys;
    int count;
    __device__ __forceinline__ bool operator()(int token) const {
        bool found = false;
        for (int i = 0; i < count; ++i) found |= keys[i] == token;
        return found;
    }
};

// V_MODE: UNICA_B200_V_*.  Clusters: heads of K, heads of V, then eight tiles of Q each.
template <int V_MODE>
__global__ void __cluster_dims__(CALL_CLUSTER, 1, 1) __launch_bounds__(CALL_THREADS) quantize_call_int8_kernel(const __grid_constant__ CallQuantize call) {
    __shared__ CallStats sm;
    __shared__ CallOutliers outliers;
    const int rank = int(blockIdx.x) % CALL_CLUSTER, clusters_k = call.k.x ? call.heads : 0, clusters_v = call.v.x ? call.heads : 0;
    int cluster = int(blockIdx.x) / CALL_CLUSTER;
    if (cluster < clusters_k) {
        const CallOperand& op = call.k;
        const int head = cluster;
        head_stats(op.x, op.in, call.rope, NoSkip{}, head, op.n_tokens, rank, sm);
        if (rank == 0 && threadIdx.x < HEAD_DIM) op.mean[size_t(head) * HEAD_DIM + threadIdx.x] = sm.mean[threadIdx.x];
        for (int t = share(op.tiles, rank); t < share(op.tiles, rank + 1); ++t) {
            const size_t tile = size_t(head) * op.tiles + t;
            rows_int8_tile<KEY_TILE>(op.x, op.in, sm.mean, head, t, op.n_tokens, reinterpret_cast<int8_t*>(op.codes) + tile * (KEY_TILE * HEAD_DIM),
                                     static_cast<float*>(op.scales) + tile, call.rope, sm.scratch);
            __syncthreads();
        }
    } else if ((cluster -= clusters_k) < clusters_v) {
        const CallOperand& op = call.v;
        const int head = cluster;
        float* scale = static_cast<float*>(op.scales);
        auto tiles = [&](auto per_token, auto skip) {
            for (int t = share(op.tiles, rank); t < share(op.tiles, rank + 1); ++t) {
                v_int8_tile<decltype(per_token)::value>(op.x, op.in, sm.low, sm.high, skip, head, t, op.tiles, op.n_tokens, reinterpret_cast<int8_t*>(op.codes),
                                                        scale, call.v_token, sm.v_tile);
                __syncthreads();
            }
        };
        if constexpr (V_MODE == UNICA_B200_V_TOKEN) {
            tiles(std::true_type{}, NoSkip{});
        } else if constexpr (V_MODE == UNICA_B200_V_OUTLIERS) {
            find_outliers(op.x, op.in, head, op.n_tokens, call.n_outliers, rank, sm.candidates, outliers);
            const SkipKeys skip{outliers.keys, call.n_outliers};
            head_stats(op.x, op.in, RopeTable{nullptr, 0}, skip, head, op.n_tokens, rank, sm);
            tiles(std::false_type{}, skip);
            if (rank == 0) {  // the outliers' rows over the channel scales
                for (int i = threadIdx.x; i < call.n_outliers * HEAD_DIM; i += CALL_THREADS) {
                    const int o = i / HEAD_DIM, c = i % HEAD_DIM, key = outliers.keys[o];
                    const float s = fmaxf(fmaxf(sm.high[c], -sm.low[c]) * (1.0f / 127.0f), 1e-12f);
                    float x = 0.0f;
                    if (key >= 0) {
                        const __nv_bfloat16* src = op.x + op.in.offset(head, key) + c;
                        x = op.in.half ? __bfloat162float(__float2bfloat16_rn(__half2float(*reinterpret_cast<const __half*>(src)))) : __bfloat162float(*src);
                    }
                    call.outlier_rows[(size_t(head) * call.n_outliers) * HEAD_DIM + i] = __fdiv_rn(x, s);
                    if (c == 0) call.outlier_keys[size_t(head) * call.n_outliers + o] = key;
                }
            }
        } else {
            head_stats(op.x, op.in, RopeTable{nullptr, 0}, NoSkip{}, head, op.n_tokens, rank, sm);
            tiles(std::false_type{}, NoSkip{});
        }
    } else {
        cluster -= clusters_v;
        const CallOperand& op = call.q;
        const int tile = cluster * CALL_CLUSTER + rank, head = tile / op.tiles, t = tile % op.tiles;
        if (head < call.heads)
            rows_int8_tile<QUERY_TILE>(op.x, op.in, nullptr, head, t, op.n_tokens, reinterpret_cast<int8_t*>(op.codes) + size_t(tile) * (QUERY_TILE * HEAD_DIM),
                                       static_cast<float*>(op.scales) + tile, call.rope, sm.scratch);
    }
    cg::this_cluster().sync();  // nobody leaves while another block may still read its shared memory
}

// max |x - mean| of the block's values -> the outer scale of all: see nvfp4_outer_rows_kernel
__device__ __forceinline__ float outer_scale(float amax) { return fmaxf(amax * (1.0f / 2688.0f), 1e-30f); }

// Clusters: heads of K, of V, of Q.
__global__ void __cluster_dims__(CALL_CLUSTER, 1, 1) __launch_bounds__(CALL_THREADS) quantize_call_fp4_kernel(const __grid_constant__ CallQuantize call) {
    __shared__ CallStats sm;
    __shared__ float q_means[CALL_GROUPS][HEAD_DIM], q_amax;
    extern __shared__ __align__(16) uint8_t tile_smem[];  // V4Tile
    const int rank = int(blockIdx.x) % CALL_CLUSTER;
    const int kind = int(blockIdx.x) / CALL_CLUSTER / call.heads, head = int(blockIdx.x) / CALL_CLUSTER % call.heads;
    if (kind == 0) {
        const CallOperand& op = call.k;
        head_stats(op.x, op.in, call.rope, NoSkip{}, head, op.n_tokens, rank, sm);
        float amax = 0.0f;
        if (threadIdx.x < HEAD_DIM) {
            const float m = sm.mean[threadIdx.x];
            amax = fmaxf(fabsf(sm.high[threadIdx.x] - m), fabsf(sm.low[threadIdx.x] - m));
            if (rank == 0) op.mean[size_t(head) * HEAD_DIM + threadIdx.x] = m;
        }
        const float outer = outer_scale(block_max<CALL_THREADS>(amax, sm.scratch));
        if (rank == 0 && threadIdx.x == 0) op.outer[head] = outer;
        for (int t = share(op.tiles, rank); t < share(op.tiles, rank + 1); ++t) {
            const size_t tile = size_t(head) * op.tiles + t;
            rows_fp4_tile<KEY_TILE, true>(op.x, op.in, [&](int) { return sm.mean; }, outer, head, t, op.n_tokens, op.codes + tile * (KEY_TILE * HEAD_DIM / 2),
                                          static_cast<uint8_t*>(op.scales) + tile * (KEY_TILE * 8), call.rope);
        }
    } else if (kind == 1) {
        const CallOperand& op = call.v;
        head_stats(op.x, op.in, RopeTable{nullptr, 0}, NoSkip{}, head, op.n_tokens, rank, sm);
        for (int t = share(op.tiles, rank); t < share(op.tiles, rank + 1); ++t) {
            const size_t tile = size_t(head) * op.tiles + t;
            v_fp4_tile(op.x, op.in, sm.low, sm.high, head, t, op.n_tokens, op.codes + tile * (V4_ROWS * 32),
                       static_cast<uint8_t*>(op.scales) + tile * (V4_SF_WORDS * 4), op.outer + size_t(head) * HEAD_DIM, *reinterpret_cast<V4Tile*>(tile_smem));
            __syncthreads();
        }
    } else {
        // Q: a mean per group of `smooth` tokens, whole groups per block
        const CallOperand& op = call.q;
        const int groups = (op.n_tokens + call.smooth - 1) / call.smooth, per = call.smooth / CALL_BLOCK, blocks = (op.n_tokens + CALL_BLOCK - 1) / CALL_BLOCK;
        float amax = 0.0f;
        for (int g = share(groups, rank); g < share(groups, rank + 1); ++g) {
            float s = 0.0f, lo = INFINITY, hi = -INFINITY;
            const int b1 = min((g + 1) * per, blocks);
            for (int b = g * per; b < b1; ++b) {
                block_stats(op.x, op.in, call.rope, NoSkip{}, head, b, op.n_tokens, sm, sm.part[0]);
                if (threadIdx.x < HEAD_DIM)
                    s += sm.part[0][0][threadIdx.x], lo = fminf(lo, sm.part[0][1][threadIdx.x]), hi = fmaxf(hi, sm.part[0][2][threadIdx.x]);
                __syncthreads();
            }
            if (threadIdx.x < HEAD_DIM) {
                const float m = s / float(min(b1 * CALL_BLOCK, op.n_tokens) - g * call.smooth);
                amax = fmaxf(amax, fmaxf(fabsf(hi - m), fabsf(lo - m)));
                __stcg(op.mean + (size_t(head) * groups + g) * HEAD_DIM + threadIdx.x, m);
            }
        }
        amax = block_max<CALL_THREADS>(amax, sm.scratch);
        if (threadIdx.x == 0) q_amax = amax;
        __threadfence();
        cg::this_cluster().sync();
        amax = 0.0f;
        for (int r = 0; r < CALL_CLUSTER; ++r) amax = fmaxf(amax, *cg::this_cluster().map_shared_rank(&q_amax, r));
        const float outer = outer_scale(amax);
        if (rank == 0 && threadIdx.x == 0) op.outer[head] = outer;
        const int t0 = share(op.tiles, rank), t1 = share(op.tiles, rank + 1), g0 = t0 * QUERY_TILE / call.smooth;
        const int touched = t1 > t0 ? min((t1 * QUERY_TILE - 1) / call.smooth, groups - 1) - g0 + 1 : 0;  // groups of this block's tiles (its last ones may lie past the end)
        for (int i = threadIdx.x; i < touched * HEAD_DIM; i += CALL_THREADS)
            q_means[i / HEAD_DIM][i % HEAD_DIM] = __ldcg(op.mean + (size_t(head) * groups + g0) * HEAD_DIM + i);
        __syncthreads();
        for (int t = t0; t < t1; ++t) {
            const size_t tile = size_t(head) * op.tiles + t;
            rows_fp4_tile<QUERY_TILE, false>(op.x, op.in, [&](int token) { return q_means[token / call.smooth - g0]; }, outer, head, t, op.n_tokens,
                                             op.codes + tile * (QUERY_TILE * HEAD_DIM / 2), static_cast<uint8_t*>(op.scales) + tile * (QUERY_TILE * 8), call.rope);
        }
    }
    cg::this_cluster().sync();
}

int quantize_call_int8(const CallQuantize& call, cudaStream_t stream) {
    if (int e = unica_check_device()) return e;
    const long long q_tiles = call.q.x ? (static_cast<long long>(call.heads) * call.q.tiles + CALL_CLUSTER - 1) / CALL_CLUSTER : 0;
    const long long clusters = (call.k.x ? call.heads : 0) + (call.v.x ? call.heads : 0) + q_tiles;
    if (clusters > (1 << 27)) return unica_fail(UNICA_B200_ERR_ARGUMENT, "quantize_call: too many heads and tiles");
    const dim3 grid(unsigned(clusters) * CALL_CLUSTER);
    if (call.v_mode == UNICA_B200_V_TOKEN)
        quantize_call_int8_kernel<UNICA_B200_V_TOKEN><<<grid, CALL_THREADS, 0, stream>>>(call);
    else if (call.v_mode == UNICA_B200_V_OUTLIERS)
        quantize_call_int8_kernel<UNICA_B200_V_OUTLIERS><<<grid, CALL_THREADS, 0, stream>>>(call);
    else
        quantize_call_int8_kernel<UNICA_B200_V_CHANNEL><<<grid, CALL_THREADS, 0, stream>>>(call);
    return unica_check_launch("quantize_call_int8");
}

int quantize_call_fp4(const CallQuantize& call, cudaStream_t stream) {
    if (int e = unica_check_device()) return e;
    constexpr int SMEM = int(sizeof(V4Tile));
    static_assert(SMEM + sizeof(CallStats) + CALL_GROUPS * HEAD_DIM * 4 <= 99 * 1024, "two blocks per SM");
    if (cudaFuncSetAttribute(quantize_call_fp4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)
        return unica_check_launch("quantize_call_fp4 (shared memory size)");
    quantize_call_fp4_kernel<<<dim3(3u * call.heads * CALL_CLUSTER), CALL_THREADS, SMEM, stream>>>(call);
    return unica_check_launch("quantize_call_fp4");
}

}  // namespace unica

// The quantization of a short call (up to CALL_TOKENS tokens) in ONE launch: Q, K and V of all heads, statistics included.
//
// The separate passes need three to eight launches for this, each a few microseconds on the device and as many on the host:
// for 4 heads x 1024 tokens that was most of the call.  Here the grid is made of clusters of eight blocks (four for short heads, see the host code), each of which is
// given a head's K, a head's V or (NVFP4) a head's Q, and in INT8 eight tiles of Q, which need no statistics:
//   1. the blocks of a cluster take the statistics of an eighth of the head's 256-token blocks each,
//   2. they read one another's partial results through distributed shared memory, all in the same order,
//   3. and quantize an eighth of the head's tiles each; the tokens come out of L2 now.
// What bounds it: latency.  For few tokens two dependent trips to memory and a cluster barrier each way; at 30 heads x 4128 tokens every
// block alternates between loads and conversions: with three blocks per SM a third of the chip's warps were in flight and issue 37 % busy, with four it
// is 47 and 43 %.  So where there are blocks enough, four share an SM in INT8 (64 registers, some 110 bytes of them spilled in bfloat16; the clusters of K and V of that size are then on the GPU together) and
// three in NVFP4 and rotated (80 registers; rotated rows spill 130 to 180 bytes), with nothing loaded ahead of a tile, which the other blocks make
// up for: a call of 30 x 4128 per token 376.8 -> 370.3 us, with outliers 381.7 -> 363.0.  Where there are not (AHEAD, see quantize_call_int8 and
// quantize_call_fp4), a block has more registers, the next tile under way while it works on one, and rotated twice the tokens in flight in the
// statistics.  Minima and maxima are taken on bfloat16 pairs, and outliers are looked for by all warps.
//
// Sums run in the order of channel_stats_kernel and its finish kernel (quantize.cu), minima and maxima are exact: the
// operands are bit for bit those of the separate passes.
#include <cooperative_groups.h>

#include <atomic>
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
        V4Tile v4_tile[2];
        VTileSmem v_tile[2];                                               // tiles of V on their way round
        unsigned long long candidates[CALL_TOKENS / CALL_CLUSTER + 1];  // the block's tokens, see find_outliers
    };
    float mean[HEAD_DIM], low[HEAD_DIM], high[HEAD_DIM];
    float scratch[2][CALL_THREADS / 32];  // by turns, so that a tile's maximum does not have to wait for the last one's readers
};
// this block's share of `count` things
template <int CLUSTER = CALL_CLUSTER>
__device__ __forceinline__ int share(int count, int rank) { return count * rank / CLUSTER; }

// Sum, min and max per channel of 256-token block `b` into out[3][128]: channel_stats_kernel's arithmetic.
template <bool SUMS, bool RANGE, int LOADS, typename Skip>
__device__ __forceinline__ void block_stats(const __nv_bfloat16* __restrict__ x, const TokenLayout& in, const RopeTable& rope, Skip skip, int head, int b,
                                            int n_tokens, CallStats& sm, float (&out)[3][HEAD_DIM]) {
    const int chunk = threadIdx.x % 16, lane = threadIdx.x / 16;
    float2 sum[4], low[4], high[4];
    // minima and maxima of values that are not rotated are taken on the bfloat16 pairs as they come (exact)
    const bool packed = !rope.table;
    __nv_bfloat162 low2[4], high2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sum[i] = make_float2(0.0f, 0.0f), low[i] = make_float2(INFINITY, INFINITY), high[i] = make_float2(-INFINITY, -INFINITY);
        low2[i] = __floats2bfloat162_rn(INFINITY, INFINITY), high2[i] = __floats2bfloat162_rn(-INFINITY, -INFINITY);
    }
    const int first = b * CALL_BLOCK + lane;
    const __nv_bfloat16* src = x + in.offset(head, 0) + chunk * 8;
#pragma unroll
    for (int part = 0; part < CALL_BLOCK / CALL_LANES; part += LOADS) {  // so many loads in flight
        uint4 raw[LOADS], turns[LOADS];
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int token = first + (part + j) * CALL_LANES;
            raw[j] = turns[j] = make_uint4(0, 0, 0, 0);
            if (token < n_tokens) {
                raw[j] = load_bf16x8(src + token * in.token, in.half);
                if (rope.table) turns[j] = *reinterpret_cast<const uint4*>(rope.row(in, head, token) + chunk * 8);
            }
        }
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int token = first + (part + j) * CALL_LANES;
            if (token >= n_tokens || skip(token)) continue;
            float2 v[4];
            unpack8(raw[j], v);
            if (rope.table) rope8(*reinterpret_cast<float(*)[8]>(v), turns[j]);
            const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (SUMS) sum[i] = add2(sum[i], v[i]);
                if (RANGE && packed) low2[i] = __hmin2(low2[i], pairs[i]), high2[i] = __hmax2(high2[i], pairs[i]);
                if (RANGE && !packed) {
                    low[i] = make_float2(fminf(low[i].x, v[i].x), fminf(low[i].y, v[i].y));
                    high[i] = make_float2(fmaxf(high[i].x, v[i].x), fmaxf(high[i].y, v[i].y));
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (SUMS) *reinterpret_cast<float2*>(&sm.lanes[0][lane][chunk * 8 + 2 * i]) = sum[i];
        if (RANGE) {
            if (packed) low[i] = __bfloat1622float2(low2[i]), high[i] = __bfloat1622float2(high2[i]);
            *reinterpret_cast<float2*>(&sm.lanes[1][lane][chunk * 8 + 2 * i]) = low[i];
            *reinterpret_cast<float2*>(&sm.lanes[2][lane][chunk * 8 + 2 * i]) = high[i];
        }
    }
    __syncthreads();
    if (threadIdx.x < HEAD_DIM) {
        float s = 0.0f, lo = INFINITY, hi = -INFINITY;
#pragma unroll
        for (int l = 0; l < CALL_LANES; ++l) {
            if (SUMS) s += sm.lanes[0][l][threadIdx.x];
            if (RANGE) lo = fminf(lo, sm.lanes[1][l][threadIdx.x]), hi = fmaxf(hi, sm.lanes[2][l][threadIdx.x]);
        }
        if (SUMS) out[0][threadIdx.x] = s;
        if (RANGE) out[1][threadIdx.x] = lo, out[2][threadIdx.x] = hi;
    }
    __syncthreads();
}

// The head's mean (SUMS), min and max (RANGE) into sm of every block of the cluster.  Every thread of the cluster calls it.
template <bool SUMS, bool RANGE, int CLUSTER = CALL_CLUSTER, int LOADS = 8, typename Skip>
__device__ __forceinline__ void head_stats(const __nv_bfloat16* __restrict__ x, const TokenLayout& in, const RopeTable& rope, Skip skip, int head,
                                           int n_tokens, int rank, CallStats& sm) {
    const int blocks = (n_tokens + CALL_BLOCK - 1) / CALL_BLOCK, b0 = share<CLUSTER>(blocks, rank), b1 = share<CLUSTER>(blocks, rank + 1);
    for (int b = b0; b < b1; ++b) block_stats<SUMS, RANGE, LOADS>(x, in, rope, skip, head, b, n_tokens, sm, sm.part[b - b0]);
    cg::this_cluster().sync();
    if (threadIdx.x < HEAD_DIM) {
        // all blocks' partial results asked for before the first is added up: a trip to another SM takes some hundred cycles
        float s = 0.0f, lo = INFINITY, hi = -INFINITY;
        float theirs_s[CLUSTER], theirs_lo[CLUSTER], theirs_hi[CLUSTER];
        const int most = (blocks + CLUSTER - 1) / CLUSTER;
        if (most == 1) {
#pragma unroll
            for (int r = 0; r < CLUSTER; ++r) {
                const CallStats* theirs = cg::this_cluster().map_shared_rank(&sm, r);
                if (SUMS) theirs_s[r] = theirs->part[0][0][threadIdx.x];
                if (RANGE) theirs_lo[r] = theirs->part[0][1][threadIdx.x], theirs_hi[r] = theirs->part[0][2][threadIdx.x];
            }
#pragma unroll
            for (int r = 0; r < CLUSTER; ++r)
                if (share<CLUSTER>(blocks, r + 1) > share<CLUSTER>(blocks, r)) {  // the others hold nothing
                    if (SUMS) s += theirs_s[r];
                    if (RANGE) lo = fminf(lo, theirs_lo[r]), hi = fmaxf(hi, theirs_hi[r]);
                }
        } else {
#pragma unroll
            for (int r = 0; r < CLUSTER; ++r) {
                const CallStats* theirs = cg::this_cluster().map_shared_rank(&sm, r);
                const int parts = share<CLUSTER>(blocks, r + 1) - share<CLUSTER>(blocks, r);
                float part_s[CALL_PARTS], part_lo[CALL_PARTS], part_hi[CALL_PARTS];
#pragma unroll
                for (int i = 0; i < CALL_PARTS; ++i) {
                    if (SUMS) part_s[i] = theirs->part[i][0][threadIdx.x];
                    if (RANGE) part_lo[i] = theirs->part[i][1][threadIdx.x], part_hi[i] = theirs->part[i][2][threadIdx.x];
                }
#pragma unroll
                for (int i = 0; i < CALL_PARTS; ++i)
                    if (i < parts) {
                        if (SUMS) s += part_s[i];
                        if (RANGE) lo = fminf(lo, part_lo[i]), hi = fmaxf(hi, part_hi[i]);
                    }
            }
        }
        if (SUMS) sm.mean[threadIdx.x] = s / float(n_tokens);
        if (RANGE) sm.low[threadIdx.x] = lo, sm.high[threadIdx.x] = hi;
    }
    __syncthreads();
}

// The n_outliers keys with the largest max |v| of the head, ties to the lower key (what the reference's emulation takes), NaN above
// all numbers (as torch's topk has it), in every block of the cluster: -1 where the head has fewer keys.  Every warp picks the largest of an eighth of the block's
// tokens, then one warp per block picks among all blocks' picks.
constexpr int CALL_WARPS = CALL_THREADS / 32, CALL_PICKS = CALL_WARPS * CALL_OUTLIERS;
struct CallOutliers {
    unsigned long long mine[CALL_PICKS];  // this block's picks: max |v| as bits, then the complement of the key; 0: none
    int keys[CALL_OUTLIERS];
    uint32_t is_outlier[CALL_TOKENS / 32];  // a bit per token of the head
};
__device__ __forceinline__ unsigned long long larger(unsigned long long a, unsigned long long b) { return a > b ? a : b; }
__device__ __forceinline__ unsigned long long warp_largest(unsigned long long x) {
#pragma unroll
    for (int d = 16; d > 0; d /= 2) x = larger(x, __shfl_xor_sync(0xffffffffu, x, d));
    return x;
}
// the `count` largest of a warp's values (N per lane), one after the other
template <int N, typename Take>
__device__ __forceinline__ void take_largest(unsigned long long (&value)[N], int count, Take take) {
    for (int o = 0; o < count; ++o) {
        unsigned long long best = value[0];
#pragma unroll
        for (int j = 1; j < N; ++j) best = larger(best, value[j]);
        best = warp_largest(best);
        take(o, best);
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (value[j] == best) value[j] = 0;
    }
}
__device__ __forceinline__ void find_outliers(const __nv_bfloat16* __restrict__ v, const TokenLayout& in, int head, int n_tokens, int n_outliers, int rank,
                                              unsigned long long* candidates, CallOutliers& sm) {
    const int t0 = share(n_tokens, rank), count = share(n_tokens, rank + 1) - t0;
    const int chunk = threadIdx.x % 16, lane = threadIdx.x / 16;
    for (int i = threadIdx.x; i < CALL_TOKENS / 32; i += CALL_THREADS) sm.is_outlier[i] = 0;
    const __nv_bfloat16* first = v + in.offset(head, t0) + chunk * 8;
    for (int i0 = 0; i0 < count; i0 += 8 * CALL_LANES) {  // eight loads in flight
        uint4 raw[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = i0 + j * CALL_LANES + lane;
            raw[j] = i < count ? load_bf16x8(first + i * in.token, in.half) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = i0 + j * CALL_LANES + lane;
            const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
            const __nv_bfloat162 top = __hmax2_nan(__hmax2_nan(__habs2(pairs[0]), __habs2(pairs[1])), __hmax2_nan(__habs2(pairs[2]), __habs2(pairs[3])));
            const float2 two = __bfloat1622float2(top);
            unsigned amax = max(__float_as_uint(two.x), __float_as_uint(two.y));  // (the bits of non-negative floats are in their order)
#pragma unroll
            for (int d = 8; d > 0; d /= 2) amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, d));
            if (chunk == 0 && i < count) candidates[i] = (static_cast<unsigned long long>(amax) << 32) | (0xffffffffu - unsigned(t0 + i));
        }
    }
    __syncthreads();
    {
        unsigned long long value[CALL_TOKENS / CALL_CLUSTER / CALL_THREADS + 1];
#pragma unroll
        for (int j = 0; j < CALL_TOKENS / CALL_CLUSTER / CALL_THREADS + 1; ++j) {
            const int i = j * CALL_THREADS + threadIdx.x;
            value[j] = i < count ? candidates[i] : 0;
        }
        take_largest(value, n_outliers, [&](int o, unsigned long long best) {
            if (threadIdx.x % 32 == 0) sm.mine[threadIdx.x / 32 * CALL_OUTLIERS + o] = best;
        });
    }
    cg::this_cluster().sync();
    if (threadIdx.x < 32) {
        constexpr int PER_LANE = CALL_CLUSTER * CALL_PICKS / 32;
        unsigned long long value[PER_LANE];
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) {  // lanes side by side on one block's picks
            const int i = j * 32 + threadIdx.x;
            value[j] = i % CALL_OUTLIERS < n_outliers ? cg::this_cluster().map_shared_rank(&sm, i / CALL_PICKS)->mine[i % CALL_PICKS] : 0;
        }
        take_largest(value, n_outliers, [&](int o, unsigned long long best) {
            if (threadIdx.x == 0) {
                const int key = best ? int(0xffffffffu - unsigned(best)) : -1;
                sm.keys[o] = key;
                if (key >= 0) sm.is_outlier[key / 32] |= 1u << (key % 32);
            }
        });
    }
    __syncthreads();
}

struct NoSkip {
    __device__ __forceinline__ bool operator()(int) const { return false; }
};
struct SkipKeys {
    const uint32_t* is_outlier;
    __device__ __forceinline__ bool operator()(int token) const { return (is_outlier[token / 32] >> (token % 32)) & 1; }
};

// Tiles first .. last - 1 in order; AHEAD: each loaded while the one before is worked on.
template <bool AHEAD, typename Raw, typename Load, typename Finish>
__device__ __forceinline__ void each_tile(int first, int last, Load load, Finish finish) {
    if constexpr (AHEAD) {
        if (first >= last) return;
        Raw raw, next;
        load(raw, first);
        for (int t = first; t < last; ++t) {
            if (t + 1 < last) load(next, t + 1);
            finish(raw, t);
            raw = next;
        }
    } else {
        for (int t = first; t < last; ++t) {
            Raw raw;
            load(raw, t);
            finish(raw, t);
        }
    }
}

// The kernel is launched to overlap the end of the kernel before it in the stream, whatever that is: its blocks are set up while that one's
// results are being written back (a loop of 4 heads x 1024 tokens 24.7 -> 22.7 us a call, 2 x 8 x 1000 queries with 77 keys 22.6 -> 20.4).
// Nothing is read or written before the wait: the addresses of all that is read follow from a head or a pointer that comes out of behind_wait
// (in INT8 from the head: with q's, k's and v's pointers, as in NVFP4, calls of 1 head x 8192 tokens per channel took 106.6 us, not 103.4).  And the call's next
// kernel is let in only after it, for two reasons: its blocks take tensor memory, which a kernel before the call may not have taken yet; and
// smooth_bias_few_kernel reads K before a wait of its own, which is as early as K is sure to be there.
__device__ __forceinline__ void begin_call() {
    wait_for_previous_kernel();
    let_next_kernel_start();
}
// Not so for INT8 in a captured call: replayed one after the other, such calls are faster in the usual order (4 x 1500 31.1 -> 29.0 us, 10 x 300
// 21.0 -> 19.2, up to 4 x 500 0.2 us slower; NVFP4 1 x 500 27.5 against 25.6).
static bool capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus state = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &state) == cudaSuccess) return state != cudaStreamCaptureStatusNone;
    cudaGetLastError();  // (the null stream while another one captures: the launch will say so)
    return false;
}

// V_MODE: UNICA_B200_V_*; HALF, ROPE: the input is float16, Q and K are rotated (template parameters so that the other calls
// carry none of it); AHEAD: see each_tile.  Clusters: heads of K, heads of V, then CLUSTER tiles of Q each.
template <int V_MODE, bool HALF, bool ROPE, int CLUSTER, bool AHEAD>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(CALL_THREADS, ROPE || AHEAD ? 3 : 4) quantize_call_int8_kernel(const __grid_constant__ CallQuantize call) {
    begin_call();
    __shared__ CallStats sm;
    __shared__ CallOutliers outliers;
    const RopeTable rope = ROPE ? call.rope : RopeTable{nullptr, 0}, none{nullptr, 0};
    const int rank = int(blockIdx.x) % CLUSTER, clusters_k = call.k.x ? call.heads : 0, clusters_v = call.v.x ? call.heads : 0;
    int cluster = int(blockIdx.x) / CLUSTER;
    if (cluster < clusters_k) {
        const CallOperand& op = call.k;
        TokenLayout in = op.in;
        in.half = HALF;
        const int head = behind_wait(cluster);
        head_stats<true, false, CLUSTER, ROPE ? 4 : 8>(op.x, in, rope, NoSkip{}, head, op.n_tokens, rank, sm);
        if (rank == 0 && threadIdx.x < HEAD_DIM) op.mean[size_t(head) * HEAD_DIM + threadIdx.x] = sm.mean[threadIdx.x];
        each_tile<AHEAD, RowsRaw<KEY_TILE>>(
            share<CLUSTER>(op.tiles, rank), share<CLUSTER>(op.tiles, rank + 1),
            [&](auto& raw, int t) { rows_load<KEY_TILE, CALL_THREADS, ROPE>(raw, op.x, in, head, t, op.n_tokens); },
            [&](const auto& raw, int t) {
                const size_t tile = size_t(head) * op.tiles + t;
                rows_int8_finish<KEY_TILE, CALL_THREADS, ROPE>(raw, in, sm.mean, head, t, op.n_tokens, reinterpret_cast<int8_t*>(op.codes) + tile * (KEY_TILE * HEAD_DIM),
                                                               static_cast<float*>(op.scales) + tile, rope, sm.scratch[t & 1]);
            });
    } else if ((cluster -= clusters_k) < clusters_v) {
        const CallOperand& op = call.v;
        TokenLayout in = op.in;
        in.half = HALF;
        constexpr bool OUTLIERS = V_MODE == UNICA_B200_V_OUTLIERS;  // (of the two, what costs them less: 1 x 1024 33.7 us a call with the head, 33.0 with the pointer)
        const __nv_bfloat16* x = OUTLIERS ? behind_wait(op.x) : op.x;
        const int head = OUTLIERS ? cluster : behind_wait(cluster);
        float* scale = static_cast<float*>(op.scales);
        auto tiles = [&](auto per_token, auto skip) {
            each_tile<AHEAD, VRaw>(
                share<CLUSTER>(op.tiles, rank), share<CLUSTER>(op.tiles, rank + 1), [&](auto& raw, int t) { v_load(raw, x, in, skip, head, t, op.n_tokens); },
                [&](const auto& raw, int t) {
                    v_int8_finish<decltype(per_token)::value>(raw, sm.low, sm.high, head, t, op.tiles, op.n_tokens, reinterpret_cast<int8_t*>(op.codes), scale,
                                                              call.v_token, sm.v_tile[t & 1]);
                });
        };
        if constexpr (V_MODE == UNICA_B200_V_TOKEN) {
            tiles(std::true_type{}, NoSkip{});
        } else if constexpr (V_MODE == UNICA_B200_V_OUTLIERS) {
            find_outliers(x, in, head, op.n_tokens, call.n_outliers, rank, sm.candidates, outliers);
            const SkipKeys skip{outliers.is_outlier};
            head_stats<false, true, CLUSTER>(x, in, none, skip, head, op.n_tokens, rank, sm);
            tiles(std::false_type{}, skip);
            if (rank == 0) {  // the outliers' rows over the channel scales
                for (int i = threadIdx.x; i < call.n_outliers * HEAD_DIM; i += CALL_THREADS) {
                    const int o = i / HEAD_DIM, c = i % HEAD_DIM, key = outliers.keys[o];
                    const float s = fmaxf(fmaxf(sm.high[c], -sm.low[c]) * (1.0f / 127.0f), 1e-12f);
                    float value = 0.0f;
                    if (key >= 0) {
                        const __nv_bfloat16* src = x + in.offset(head, key) + c;
                        value = HALF ? __bfloat162float(__float2bfloat16_rn(__half2float(*reinterpret_cast<const __half*>(src)))) : __bfloat162float(*src);
                    }
                    call.outlier_rows[(size_t(head) * call.n_outliers) * HEAD_DIM + i] = __fdiv_rn(value, s);
                    if (c == 0) call.outlier_keys[size_t(head) * call.n_outliers + o] = key;
                }
            }
        } else {
            head_stats<false, true, CLUSTER>(x, in, none, NoSkip{}, head, op.n_tokens, rank, sm);
            tiles(std::false_type{}, NoSkip{});
        }
    } else {
        cluster -= clusters_v;
        const CallOperand& op = call.q;
        TokenLayout in = op.in;
        in.half = HALF;
        const int tile = behind_wait(cluster * CLUSTER + rank), head = tile / op.tiles, t = tile % op.tiles;
        if (head < call.heads) {
            int8_t* codes = reinterpret_cast<int8_t*>(op.codes) + size_t(tile) * (QUERY_TILE * HEAD_DIM);
            float* scale = static_cast<float*>(op.scales) + tile;
            if constexpr (ROPE)
                rows_int8_tile<QUERY_TILE, CALL_THREADS, true>(op.x, in, nullptr, head, t, op.n_tokens, codes, scale, rope, sm.scratch[0]);
            else
                rows_int8_tile_raw<QUERY_TILE>(op.x, in, head, t, op.n_tokens, codes, scale, sm.scratch[0]);
        }
    }
    cg::this_cluster().sync();  // nobody leaves while another block may still read its shared memory
}

// max |x - mean| of the block's values -> the outer scale of all: see nvfp4_outer_rows_kernel
__device__ __forceinline__ float outer_scale(float amax) { return fmaxf(amax * (1.0f / 2688.0f), 1e-30f); }

// HALF: the inputs are float16 (1) or bfloat16 (0), or each what its layout says.  Clusters: heads of K, of V, of Q.  Rotated inputs load their
// angles too, and without AHEAD half as many tokens at a time in the statistics, so that three blocks fit an SM (2 x 16 heads x 777 tokens: with two blocks
// and eight tokens 61.5 us a call, with three and four 56.1; with three and eight, which spills more, 59.4).
constexpr int EACH_ITS_OWN = 2;
template <int HALF, bool ROPE, int CLUSTER, bool AHEAD>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(CALL_THREADS, ROPE && AHEAD ? 2 : 3) quantize_call_fp4_kernel(const __grid_constant__ CallQuantize call) {
    begin_call();
    __shared__ CallStats sm;
    __shared__ float q_means[CALL_GROUPS][HEAD_DIM], q_amax;
    const RopeTable rope = ROPE ? call.rope : RopeTable{nullptr, 0};
    const int rank = int(blockIdx.x) % CLUSTER;
    const int kind = int(blockIdx.x) / CLUSTER / call.heads, any_head = int(blockIdx.x) / CLUSTER % call.heads;
    const int head = AHEAD ? behind_wait(any_head) : any_head;  // (of the two, what costs less: 40 x 128 28.9 us a call with the pointers, 29.9 with the head; 4 x 8192 182.1 and 179.4)
    if (kind == 0) {
        const CallOperand& op = call.k;
        const __nv_bfloat16* x = AHEAD ? op.x : behind_wait(op.x);
        TokenLayout in = op.in;
        if (HALF != EACH_ITS_OWN) in.half = HALF;
        head_stats<true, true, CLUSTER, ROPE && !AHEAD ? 4 : 8>(x, in, rope, NoSkip{}, head, op.n_tokens, rank, sm);
        float amax = 0.0f;
        if (threadIdx.x < HEAD_DIM) {
            const float m = sm.mean[threadIdx.x];
            amax = fmaxf(fabsf(sm.high[threadIdx.x] - m), fabsf(sm.low[threadIdx.x] - m));
            if (rank == 0) op.mean[size_t(head) * HEAD_DIM + threadIdx.x] = m;
        }
        const Fp4Outer outer = fp4_outer(outer_scale(block_max<CALL_THREADS>(amax, sm.scratch[0])));
        if (rank == 0 && threadIdx.x == 0) op.outer[head] = outer.value;
        for (int t = share<CLUSTER>(op.tiles, rank); t < share<CLUSTER>(op.tiles, rank + 1); ++t) {  // (no barrier in a tile: the warps run ahead of one another)
            const size_t tile = size_t(head) * op.tiles + t;
            rows_fp4_tile<KEY_TILE, true, ROPE>(x, in, [&](int) { return sm.mean; }, outer, head, t, op.n_tokens, op.codes + tile * (KEY_TILE * HEAD_DIM / 2),
                                          static_cast<uint8_t*>(op.scales) + tile * (KEY_TILE * 8), rope);
        }
    } else if (kind == 1) {
        const CallOperand& op = call.v;
        const __nv_bfloat16* x = AHEAD ? op.x : behind_wait(op.x);
        TokenLayout in = op.in;
        if (HALF != EACH_ITS_OWN) in.half = HALF;
        head_stats<false, true, CLUSTER>(x, in, RopeTable{nullptr, 0}, NoSkip{}, head, op.n_tokens, rank, sm);
        each_tile<AHEAD, VRaw>(
            share<CLUSTER>(op.tiles, rank), share<CLUSTER>(op.tiles, rank + 1), [&](auto& raw, int t) { v_fp4_load(raw, x, in, head, t, op.n_tokens); },
            [&](const auto& raw, int t) {
                const size_t tile = size_t(head) * op.tiles + t;
                v_fp4_finish(raw, sm.low, sm.high, t, op.codes + tile * (V4_ROWS * 32), static_cast<uint8_t*>(op.scales) + tile * (V4_SF_WORDS * 4),
                             op.outer + size_t(head) * HEAD_DIM, sm.v4_tile[t & 1]);
            });
    } else {
        // Q: a mean per group of `smooth` tokens, whole groups per block
        const CallOperand& op = call.q;
        const __nv_bfloat16* x = AHEAD ? op.x : behind_wait(op.x);
        TokenLayout in = op.in;
        if (HALF != EACH_ITS_OWN) in.half = HALF;
        const int groups = (op.n_tokens + call.smooth - 1) / call.smooth, per = call.smooth / CALL_BLOCK, blocks = (op.n_tokens + CALL_BLOCK - 1) / CALL_BLOCK;
        float amax = 0.0f;
        for (int g = share<CLUSTER>(groups, rank); g < share<CLUSTER>(groups, rank + 1); ++g) {
            float s = 0.0f, lo = INFINITY, hi = -INFINITY;
            const int b1 = min((g + 1) * per, blocks);
            for (int b = g * per; b < b1; ++b) {
                block_stats<true, true, ROPE && !AHEAD ? 4 : 8>(x, in, rope, NoSkip{}, head, b, op.n_tokens, sm, sm.part[0]);
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
        amax = block_max<CALL_THREADS>(amax, sm.scratch[0]);
        if (threadIdx.x == 0) q_amax = amax;
        __threadfence();
        cg::this_cluster().sync();
        amax = 0.0f;
        for (int r = 0; r < CLUSTER; ++r) amax = fmaxf(amax, *cg::this_cluster().map_shared_rank(&q_amax, r));
        const Fp4Outer outer = fp4_outer(outer_scale(amax));
        if (rank == 0 && threadIdx.x == 0) op.outer[head] = outer.value;
        const int t0 = share<CLUSTER>(op.tiles, rank), t1 = share<CLUSTER>(op.tiles, rank + 1), g0 = t0 * QUERY_TILE / call.smooth;
        const int touched = t1 > t0 ? min((t1 * QUERY_TILE - 1) / call.smooth, groups - 1) - g0 + 1 : 0;  // groups of this block's tiles (its last ones may lie past the end)
        for (int i = threadIdx.x; i < touched * HEAD_DIM; i += CALL_THREADS)
            q_means[i / HEAD_DIM][i % HEAD_DIM] = __ldcg(op.mean + (size_t(head) * groups + g0) * HEAD_DIM + i);
        __syncthreads();
        for (int t = t0; t < t1; ++t) {
            const size_t tile = size_t(head) * op.tiles + t;
            rows_fp4_tile<QUERY_TILE, false, ROPE>(x, in, [&](int token) { return q_means[token / call.smooth - g0]; }, outer, head, t, op.n_tokens,
                                             op.codes + tile * (QUERY_TILE * HEAD_DIM / 2), static_cast<uint8_t*>(op.scales) + tile * (QUERY_TILE * 8), rope);
        }
    }
    cg::this_cluster().sync();
}

// Clusters of a kernel that the device takes at once, as the runtime has it (asked once per device): fewer than the SMs would hold of single blocks, since a
// cluster lies within one group of SMs (48 of eight blocks, three to an SM, where 148 SMs make 55).
template <auto KERNEL, int CLUSTER>
int clusters_at_once() {
    constexpr int MAX_DEVICES = 64;
    static std::atomic<int> known[MAX_DEVICES];
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 0;
    int count = device < MAX_DEVICES ? known[device].load(std::memory_order_relaxed) : 0;
    if (count == 0) {
        cudaLaunchConfig_t config = {};
        cudaLaunchAttribute shape = {};
        shape.id = cudaLaunchAttributeClusterDimension, shape.val.clusterDim.x = CLUSTER, shape.val.clusterDim.y = shape.val.clusterDim.z = 1;
        config.gridDim = dim3(1024 * CLUSTER), config.blockDim = dim3(CALL_THREADS), config.attrs = &shape, config.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&count, KERNEL, &config) != cudaSuccess) return cudaGetLastError(), 0;
        if (device < MAX_DEVICES) known[device].store(count, std::memory_order_relaxed);
    }
    return count;
}

int quantize_call_int8(const CallQuantize& call, cudaStream_t stream, int* launches) {
    if (int e = unica_check_device()) return e;
    const CallOperand* operands[] = {&call.q, &call.k, &call.v};
    const CallOperand* first = nullptr;
    for (const CallOperand* op : operands) {
        if (!op->x) continue;
        if (!first) first = op;
        if (op->in.half == first->in.half) continue;
        for (const CallOperand* alone : operands) {  // element types differ: the kernel has one, so each operand alone
            if (!alone->x) continue;
            CallQuantize one = call;
            if (alone != &call.q) one.q = {};
            if (alone != &call.k) one.k = {};
            if (alone != &call.v) one.v = {};
            if (int e = quantize_call_int8(one, stream, launches)) return e;
        }
        return UNICA_B200_OK;
    }
    const long long q_tiles = call.q.x ? static_cast<long long>(call.heads) * call.q.tiles : 0, kv_heads = (call.k.x ? call.heads : 0) + (call.v.x ? call.heads : 0);
    int sms = 0;
    if (int e = unica_sm_count(&sms)) return e;
    const int keys = call.k.n_tokens > call.v.n_tokens ? call.k.n_tokens : call.v.n_tokens;  // (a call may have one of the two alone)
    const bool rotated = call.rope.table, outliers = call.v_mode == UNICA_B200_V_OUTLIERS;
    // Four blocks per head, as in quantize_call_fp4, where eight would crowd the SMs.  How much they may depends on what a second wave costs and on what the four then
    // have to do: up to 512 keys 3.7 to an SM (36 x 300 25.7 -> 22.1 us a call; 32 x 300 23.2 against 24.4), up to 1024 3.2 (36 x 777 47.9 -> 42.9, 32 x 600 36.1 -> 33.3;
    // 28 x 1024 42.9 against 43.9), up to 2048 4 (60 x 2048 222 -> 219.7; 34 x 1500 77.2 against 81.8); rotated, up to 1024, 3 (32 x 777 47.1 against 49.5 with 4).  Up to 256
    // always, since one block has all statistics then and four have a tile each (16 x 200 19.2 -> 18.4, rotated 22.1 -> 18.8; 4 x 512 17.0 against 18.5).
    const double per_sm = double(kv_heads * CALL_CLUSTER) / sms;  // blocks for K and V, with eight to a head
    const double most = rotated ? 3 : keys <= 2 * CALL_BLOCK ? 3.7 : keys <= 4 * CALL_BLOCK ? 3.2 : 4;
    const bool four = kv_heads > 0 && !outliers && (keys <= CALL_BLOCK || (keys <= (rotated ? 4 : 8) * CALL_BLOCK && per_sm > most));
    const int cluster = four ? 4 : CALL_CLUSTER;
    if (keys > cluster * CALL_PARTS * CALL_BLOCK) return unica_fail(UNICA_B200_ERR_ARGUMENT, "quantize_call: more tokens than a cluster's blocks have room for");
    const long long clusters = kv_heads + (q_tiles + cluster - 1) / cluster;
    if (clusters > (1 << 27)) return unica_fail(UNICA_B200_ERR_ARGUMENT, "quantize_call: too many heads and tiles");
    const dim3 grid(unsigned(clusters) * cluster);
    // Loads ahead of a tile, with three blocks per SM, or four blocks per SM without.  Ahead where a block has several tiles and at most one other block
    // beside it (1 x 8192 per token 123.5 -> 121.3 us a call, 4 x 4128 73.6 -> 71.3; 24 x 1024 44.9 against 46.5).  With outliers, whose V takes longest, what matters is that Q's tiles do
    // not get in between: three blocks per SM where that has room for K and V but not for Q beside them (20 x 777 42.7 -> 40.3, 16 x 4128 217 -> 212; 8 x 2048 53.1
    // against 54.0, 28 x 2048 130.6 against 139.8).
    const int room = outliers ? clusters_at_once<quantize_call_int8_kernel<UNICA_B200_V_OUTLIERS, false, false, CALL_CLUSTER, true>, CALL_CLUSTER>() : 0;
    const bool ahead = !rotated && (outliers ? kv_heads <= room && clusters > room : keys > cluster * KEY_TILE && kv_heads * cluster <= 2 * sms);
    auto launch = [&](auto half, auto rope, auto ahead) {
        constexpr bool HALF = decltype(half)::value, ROPE = decltype(rope)::value, AHEAD = decltype(ahead)::value;
        auto kernel = call.v_mode == UNICA_B200_V_OUTLIERS ? quantize_call_int8_kernel<UNICA_B200_V_OUTLIERS, HALF, ROPE, CALL_CLUSTER, AHEAD>
                      : call.v_mode == UNICA_B200_V_TOKEN ? (four ? quantize_call_int8_kernel<UNICA_B200_V_TOKEN, HALF, ROPE, 4, AHEAD>
                                                                  : quantize_call_int8_kernel<UNICA_B200_V_TOKEN, HALF, ROPE, CALL_CLUSTER, AHEAD>)
                                                          : (four ? quantize_call_int8_kernel<UNICA_B200_V_CHANNEL, HALF, ROPE, 4, AHEAD>
                                                                  : quantize_call_int8_kernel<UNICA_B200_V_CHANNEL, HALF, ROPE, CALL_CLUSTER, AHEAD>);
        launch_after(kernel, grid, CALL_THREADS, 0, stream, !capturing(stream), call);
    };
    const bool half = first->in.half;
    if (launches) ++*launches;
    const std::true_type yes{};
    const std::false_type no{};
    if (rotated)
        half ? launch(yes, yes, no) : launch(no, yes, no);
    else if (ahead)
        half ? launch(yes, no, yes) : launch(no, no, yes);
    else
        half ? launch(yes, no, no) : launch(no, no, no);
    return unica_check_launch("quantize_call_int8");
}

int quantize_call_fp4(const CallQuantize& call, cudaStream_t stream) {
    if (int e = unica_check_device()) return e;
    // Four blocks per head where a head's statistics are eight 256-token blocks at most (rotated: four), if eight blocks per head are more than
    // the chip takes at once: some of the eight have little to do in the first step, and a second wave costs its latency again
    // (2 x 16 heads x 777 tokens, rotated: 41.7 -> 38 us, 40 x 1024 not rotated 37 -> 30; calls of 20 x 2048 119.2 -> 113.3, 40 x 2048
    // 185 -> 177.3, 18 x 777, rotated, 53.7 -> 44.1; 16 x 777, rotated, which eight blocks per head do fit, 44.3 against 45.0).  Longer heads are better with eight
    // (20 x 4128, rotated, 296.8 against 304.5; not rotated the same).
    const int longest = call.q.n_tokens > call.k.n_tokens ? call.q.n_tokens : call.k.n_tokens;
    const bool rotated = call.rope.table, mixed = call.k.in.half != call.q.in.half || call.v.in.half != call.q.in.half;
    const long long clusters = 3LL * call.heads;
    // And up to 512 tokens in any case (4 x 256 21.8 -> 20.4, 12 x 500 32.5 -> 30.9, rotated 12 x 200 32.7 -> 30.8; 4 x 512 the same).
    const bool crowded = clusters > clusters_at_once<quantize_call_fp4_kernel<false, true, CALL_CLUSTER, false>, CALL_CLUSTER>();  // (three blocks per SM, rotated or not)
    const bool four = !mixed && longest <= (!crowded ? 2 : rotated ? 4 : 8) * CALL_BLOCK;
    // Rotated: with eight tokens at a time and V's loads ahead of a tile, which takes two blocks per SM, where that holds all of them at once (1 x 8192 137 -> 130 us a call, 10 x 1024
    // 47.3 -> 42.8, 23 x 777 52.4 -> 48.2; 12 x 1024 48.1 against 51.4).  Up to 512 tokens also where it takes two rounds and three blocks per SM would take
    // more than one and a tenth (40 x 500 54.9 -> 50.5, 47 x 300 47.3 -> 43.1; 36 x 300 41.8 against 42.3, 44 x 1024 94.4 against 99.2).  Not rotated: V's loads ahead cost no room, and pay
    // with more than eight tiles to a block (12 x 8192 469.5 -> 465).
    bool ahead = longest > 8 * KEY_TILE * CALL_CLUSTER;
    if (rotated && four) {
        const int two = clusters_at_once<quantize_call_fp4_kernel<false, true, 4, true>, 4>(), three = clusters_at_once<quantize_call_fp4_kernel<false, true, 4, false>, 4>();
        ahead = clusters <= two || (longest <= 2 * CALL_BLOCK && clusters <= 2 * two && 10 * clusters > 11 * three);
    } else if (rotated) {
        ahead = clusters <= clusters_at_once<quantize_call_fp4_kernel<false, true, CALL_CLUSTER, true>, CALL_CLUSTER>();
    }
    auto launch = [&](auto half, auto rope, auto ahead) {
        constexpr bool HALF = decltype(half)::value, ROPE = decltype(rope)::value, AHEAD = decltype(ahead)::value;
        auto kernel = mixed ? quantize_call_fp4_kernel<EACH_ITS_OWN, ROPE, CALL_CLUSTER, AHEAD>
                      : four ? quantize_call_fp4_kernel<HALF, ROPE, 4, AHEAD> : quantize_call_fp4_kernel<HALF, ROPE, CALL_CLUSTER, AHEAD>;
        launch_after(kernel, dim3(unsigned(clusters) * (four ? 4 : CALL_CLUSTER)), CALL_THREADS, 0, stream, true, call);
    };
    auto launch_half = [&](auto half, auto rope) { ahead ? launch(half, rope, std::true_type{}) : launch(half, rope, std::false_type{}); };
    const std::true_type yes{};
    const std::false_type no{};
    rotated ? (call.q.in.half ? launch_half(yes, yes) : launch_half(no, yes)) : (call.q.in.half ? launch_half(yes, no) : launch_half(no, no));
    return unica_check_launch("quantize_call_fp4");
}

}  // namespace unica

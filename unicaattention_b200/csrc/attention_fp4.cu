// The fast mode's flash-attention loop on tcgen05 (replaces the reference's attention_fp4, csrc/flash.cu:1380-1524).
//
// Both contractions run as tcgen05.mma kind::mxf4nvf4.block_scale.scale_vec::4X (e2m1 codes, one ue4m3 scale per 16
// elements of the contraction, FP32 accumulators in tensor memory):
//   S[t]  = Q4[t] . K4(g)^T     128 x 64,  2 instructions of K = 64 channels
//   O[t] += P4[t](g) . V4(g)    128 x 144, 1 instruction of K = 64 keys; columns 0..127 are the output channels, column
//                               128 multiplies P by a row of ones: the running softmax denominator, rescaled with O
//
// Persistent blocks, one per SM, each taking pairs of query tiles (items) blockIdx.x, blockIdx.x + gridDim.x, ...; the two
// tiles of an item (t = 0, 1) share every K and V tile.  Where pairs would leave SMs idle an item is one query tile (TILES 1: two
// softmax warpgroups, with as many registers as they like).  Key tiles are counted across items (g), and every ring runs on from
// one item to the next.  Five warpgroups:
//
//   softmax [t][w]  query tile t, key tiles g with g & 1 = w: a thread is a query row (a tensor-memory lane), all 64 scores of
//                   a tile in its registers.  The running maximum goes from one warpgroup of a query tile to the other through
//                   shared memory as soon as it is known, long before the exponentials are done, so that the two overlap: four
//                   computing warps per scheduler, against two with one warpgroup per query tile.
//   service         four warps: the scores' instructions of both query tiles; P.V of query tile 0; of 1; all copies.  They bring K's, Q's, V's and P's scale bytes into tensor memory as well.
//
// Hand-overs between warps are named barriers (see attention_int8.cu for why); what the copies and the tensor core complete
// is waited for on mbarriers, asked for ahead of time where it can be.
//
// What bounds it: issue slots and the exponential unit together.  A warp's tile is some 520 instructions of which 96 packed FP32
// ones issue for two cycles, and 69 exponentials of 8 cycles: 825 cycles per 128 x 64 tile at 37 x 8192 tokens (0.97 ms), where
// the exponential unit alone would take 552; with one warpgroup per query tile and a block per item it was 1115 (1.34 ms).  Half
// of the warps' tiles rescale O there (any of 32 rows moving its maximum makes its warp do it), a fifth at 32760.
//
// Numerics (bench/emulate.py:298-369 with the fast contract): scores x = S * (q_outer k_outer log2(e)/sqrt(d)) + bias,
// bias the exact q_mean . (k - k_mean) term of Q smoothing; running maximum m; P = 1024 * 2^(x - m) in NVFP4 along the
// keys of the tile in slot order with a fixed outer scale of 1: per 16 slots sp = e4m3(max P / 6), codes e2m1(P / sp),
// P / sp taken as 2^(x - m + 10 - log2 sp) in one ex2.approx; O = O * 2^(m_old - m) + P^ . V^; out = O / (sum of P^) *
// v_outer.  A code of P can therefore land on the other side of a rounding boundary than the emulation's (P / sp is off
// by some 1e-6 relative): results agree to rounding, not bit for bit.
//
// Scale bytes live in tensor memory, row r of an operand in lane r % 32 of column r / 32 of every 32-lane quarter, copied there
// from shared memory by the thread that issues the MMA which reads them (tcgen05.cp 32x128b.warpx4: 16 bytes per lane, all four
// quarters), as the quantizers laid them out, P's as the softmax threads wrote them a moment earlier.
//
// Tensor memory per query tile (256 columns): S 0..63 | O 64..207 | SF of Q 208..215, K 216..219, P 220..223, V 224..231.
// All waits are bounded (common.cuh).
#include <cuda_fp8.h>

#include <atomic>
#include <climits>

#include "attention_common.cuh"
#include "capi.h"
#include "fp4_common.cuh"

namespace unica {

// TILES, below: query tiles of 128 rows per item, 2 (tensor memory holds two: 2 x 232 of 512 columns) or, where that leaves SMs idle, 1.
constexpr int F4_SCORES_WARP = 0, F4_PV_WARP = 1, F4_COPY_WARP = 3, F4_SOFTMAX_WARP = 4;
template <int TILES>
constexpr int F4_THREADS = (F4_SOFTMAX_WARP + 8 * TILES) * 32;
// with two query tiles the registers are dealt out: what a thread is launched with, and has after setmaxnreg
constexpr int F4_LAUNCH_REGISTERS = 96, F4_SOFTMAX_REGISTERS = 112, F4_SERVICE_REGISTERS = 32, F4_SPLIT_REGISTERS = 128 * (4 * F4_SOFTMAX_REGISTERS + F4_SERVICE_REGISTERS);
static_assert(F4_SPLIT_REGISTERS <= F4_THREADS<2> * F4_LAUNCH_REGISTERS, "the split must fit the launch");
constexpr int F4_HALF_SLOTS = KEY_TILE / 2;  // one 16-byte piece of a row of P^: two scale blocks of 16 slots
constexpr int F4_K_RING = 4, F4_V_RING = 8;  // K4 and V4 tiles in shared memory, see f4_copy_warp
constexpr int Q4_BYTES = QUERY_TILE * HEAD_DIM / 2;  // 8192
constexpr int SFQ_BYTES = 2 * QUERY_TILE * 4;        // 1024
constexpr int K4_BYTES = KEY_TILE * HEAD_DIM / 2;    // 4096
constexpr int SFK_BYTES = 2 * KEY_TILE * 4;          // 512
constexpr int V4_TILE_ROWS = 144, V4_BYTES = 2 * V4_TILE_ROWS * 16;  // 4608
constexpr int SFV_BYTES = 256 * 4;                   // 1024: two blocks of 32 lanes x 4 words
constexpr int BIAS_BYTES = KEY_TILE * 4;             // 256
constexpr int P4_BYTES = QUERY_TILE * KEY_TILE / 2;  // 4096
constexpr int F4_S = 0, F4_O = 64, F4_SFQ = 208, F4_SFK = 216, F4_SFP = 220, F4_SFV = 224;
constexpr float P_LOG2_GAIN = 10.0f;  // P is taken times 2^10: its block scales (up to 1024 / 6) stay below e4m3's 448

template <int TILES>
struct __align__(128) Fp4Smem {
    uint8_t q[2][TILES][Q4_BYTES];            // two items
    uint32_t sfq[2][TILES][2][32][4];         // scale words as tcgen05.cp takes them: [K step] lane, word row / 32
    uint8_t k[F4_K_RING][K4_BYTES];
    uint32_t sfk[F4_K_RING][32][4];           // lane, word 2 step + row / 32
    uint8_t v[F4_V_RING][V4_BYTES];
    uint32_t sfv[F4_V_RING][2][32][4];        // block 0: channel c = word c / 32 of lane c % 32; block 1: the ones rows
    float bias[F4_V_RING][KEY_TILE];
    float mask[2][KEY_TILE];                  // what is added to the scores where there is no smoothing term: zeros / -inf in the last tile's empty slots
    uint8_t p[TILES][2][P4_BYTES];
    uint32_t sfp[TILES][2][32][4];            // P's scale words: row r = word r / 32 of lane r % 32
    float m[TILES][2][QUERY_TILE];            // the running maximum after the last tile of either warpgroup
    uint8_t staged[TILES][4][32 * STAGED_PITCH];     // output rows on their way out
    float log2_e4m3[128];                     // log2 of every non-negative e4m3 byte's value; +inf for the byte 0, so that 2^(x - that) = 0
    // s_full, pv_done: [query tile][g & 1].  (One score buffer, but a barrier for either warpgroup: a warpgroup that has not yet
    // seen the first of two phases must not take a look for the second for an answer.)
    uint64_t q_full[2], k_full[F4_K_RING], v_full[F4_V_RING], s_full[TILES][2], pv_done[TILES][2], drain[1 + TILES];
    uint32_t tmem_base;
    int abort_flag;
    int alone[2 + TILES];  // zeros: a word for each warp that drains what it issued, which no other warp's wait may cut short
};
static_assert(sizeof(Fp4Smem<2>) + 128 <= 227 * 1024, "the block's shared memory");

// scores of query tile t taken: one softmax warpgroup -> the scores warp
__device__ __forceinline__ void f4_s_free_arrive(int t) { asm volatile("bar.arrive %0, 160;" ::"r"(1 + t) : "memory"); }
__device__ __forceinline__ void f4_s_free_sync(int t) { asm volatile("bar.sync %0, 160;" ::"r"(1 + t) : "memory"); }
// P^ of query tile t by warpgroup w -> its P.V warp
__device__ __forceinline__ void f4_pv_arrive(int t, int w) { asm volatile("bar.arrive %0, 160;" ::"r"(3 + 2 * t + w) : "memory"); }
__device__ __forceinline__ void f4_pv_sync(int t, int w) { asm volatile("bar.sync %0, 160;" ::"r"(3 + 2 * t + w) : "memory"); }
// the running maximum: to warpgroup w from the other one
__device__ __forceinline__ void f4_max_arrive(int t, int w) { asm volatile("bar.arrive %0, 256;" ::"r"(7 + 2 * t + w) : "memory"); }
__device__ __forceinline__ void f4_max_sync(int t, int w) { asm volatile("bar.sync %0, 256;" ::"r"(7 + 2 * t + w) : "memory"); }
// O of an item has been read: the warpgroup of its last key tile -> the P.V warp
__device__ __forceinline__ void f4_o_read_arrive(int t) { asm volatile("bar.arrive %0, 160;" ::"r"(11 + t) : "memory"); }
__device__ __forceinline__ void f4_o_read_sync(int t) { asm volatile("bar.sync %0, 160;" ::"r"(11 + t) : "memory"); }
// the staging rows of query tile t, from the warpgroup that stored an item to the other one, which stores the next
__device__ __forceinline__ void f4_staged_arrive(int t) { asm volatile("bar.arrive %0, 256;" ::"r"(13 + t) : "memory"); }
__device__ __forceinline__ void f4_staged_sync(int t) { asm volatile("bar.sync %0, 256;" ::"r"(13 + t) : "memory"); }

// the scores warp and the copy warp meet once per key tile
__device__ __forceinline__ void f4_copies_sync() { asm volatile("bar.sync 15, 64;" ::: "memory"); }

constexpr uint32_t IDESC_F4_QK = idesc_nvf4(QUERY_TILE, KEY_TILE);
constexpr uint32_t IDESC_F4_PV = idesc_nvf4(QUERY_TILE, V4_TILE_ROWS);

// eight floats -> eight e2m1 codes in one word, element i in nibble i
__device__ __forceinline__ uint32_t e2m1x8(const float2 (&v)[4]) {
    uint32_t word;
    asm("{\n\t"
        ".reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t"
        "}"
        : "=r"(word)
        : "f"(v[0].x), "f"(v[0].y), "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y));
    return word;
}

struct Fp4Args {
    const uint8_t *q4, *k4, *v4;
    const uint32_t *sfq, *sfk, *sfv;
    const float *qk_outer, *k_outer, *v_outer, *bias;
    int q_blocks, smooth_q;
    __nv_bfloat16* out;
    TokenLayout out_layout;
    PeerOutputs peers;
    int n_queries, n_keys;
    Items items;  // (pairs of) query tiles
    float scale_log2;
    uint32_t* p_words;
    int* status;
};

// ---------------------------------------------------------------------------------------------------------------------
// the service warps.  A whole converged warp executes these statements and one elected lane issues (see attention_int8.cu).

// Scale bytes from shared memory into tensor memory; ordered before the instructions the same lane issues after it.
__device__ __forceinline__ void cp_elected(uint32_t taddr, uint64_t desc) {
    asm volatile(
        "{\n\t"
        ".reg .pred e;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;\n\t"
        "}" ::"r"(taddr),
        "l"(desc)
        : "memory");
}
// S = Q4 . K4^T of one query tile, with K's scale bytes; base: the tile's tensor memory
__device__ __forceinline__ void f4_issue_scores(uint32_t base, uint64_t q_desc, uint64_t k_desc, uint64_t sfk_desc, uint64_t* full) {
    constexpr int Q_STEP = 2 * QUERY_TILE * 16 / 16, K_STEP = 2 * KEY_TILE * 16 / 16;
    asm volatile(
        "{\n\t"
        ".reg .pred e, first, acc;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "setp.ne.u32 first, 0, 0;\n\t"
        "setp.eq.u32 acc, 0, 0;\n\t"
        "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%6], %5;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %10, [%7], [%6], first;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %3, %4, %10, [%8], [%9], acc;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%11];\n\t"
        "}" ::"r"(base + F4_S),
        "l"(q_desc), "l"(k_desc), "l"(desc_at(q_desc, Q_STEP)), "l"(desc_at(k_desc, K_STEP)), "l"(sfk_desc), "r"(base + F4_SFK), "r"(base + F4_SFQ),
        "r"(base + F4_SFQ + 4), "r"(base + F4_SFK + 2), "r"(IDESC_F4_QK), "r"(smem_u32(full))
        : "memory");
}
// O (+)= P4 . V4 of one query tile, with P's and V's scale bytes; accumulate false: an item's first key tile
__device__ __forceinline__ void f4_issue_pv(uint32_t base, uint64_t p_desc, uint64_t v_desc, uint64_t sfp_desc, uint64_t sfv_desc, bool accumulate, uint64_t* done) {
    asm volatile(
        "{\n\t"
        ".reg .pred e, acc;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "setp.ne.u32 acc, %10, 0;\n\t"
        "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%6], %3;\n\t"
        "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%7], %4;\n\t"
        "@e tcgen05.cp.cta_group::1.32x128b.warpx4 [%8], %5;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %9, [%6], [%7], acc;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%11];\n\t"
        "}" ::"r"(base + F4_O),
        "l"(p_desc), "l"(v_desc), "l"(sfp_desc), "l"(sfv_desc), "l"(desc_at(sfv_desc, 32)), "r"(base + F4_SFP), "r"(base + F4_SFV), "r"(base + F4_SFV + 4),
        "r"(IDESC_F4_PV), "r"(uint32_t(accumulate)), "r"(smem_u32(done))
        : "memory");
}

// S(g) of both query tiles as soon as K4(g) has landed and the softmax of tile g - 1 has taken the scores.  A wait that gave up
// changes nothing here: instructions on whatever lies in the buffers do no harm (the result is not stored), and every hand-over
// still finds its receiver.
template <int TILES>
__device__ __forceinline__ void f4_scores_warp(Fp4Smem<TILES>& sm, const Fp4Args& a, int k_tiles, uint32_t tmem) {
    const int total = a.items.mine() * k_tiles;
    const uint64_t q_desc0 = smem_desc(smem_u32(sm.q[0][0]), QUERY_TILE * 16, 128), k_desc0 = smem_desc(smem_u32(sm.k[0]), KEY_TILE * 16, 128);
    const uint64_t sfq_desc0 = smem_desc(smem_u32(sm.sfq[0][0]), 16, 128), sfk_desc0 = smem_desc(smem_u32(sm.sfk[0]), 16, 128);
    int n = 0, t = 0;
#pragma unroll 1
    for (int g = 0; g < total; ++g) {
        if (t == 0) mbar_wait_line(&sm.q_full[slot<2>(n)], round_parity<2>(n), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        mbar_wait_line(&sm.k_full[slot<F4_K_RING>(g)], round_parity<F4_K_RING>(g), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        const uint64_t k_desc = desc_at(k_desc0, slot<F4_K_RING>(g) * (K4_BYTES / 16)), sfk_desc = desc_at(sfk_desc0, slot<F4_K_RING>(g) * (SFK_BYTES / 16));
#pragma unroll
        for (int i = 0; i < TILES; ++i) {
            if (g > 0) f4_s_free_sync(i);
            __syncwarp();
            tc_fence_after();
            const uint32_t base = tmem + 256 * i;
            if (t == 0) {  // Q's scale bytes, for the whole item
                const uint64_t sfq_desc = desc_at(sfq_desc0, (slot<2>(n) * TILES + i) * (SFQ_BYTES / 16));
                cp_elected(base + F4_SFQ, sfq_desc);
                cp_elected(base + F4_SFQ + 4, desc_at(sfq_desc, SFQ_BYTES / 32));
            }
            f4_issue_scores(base, desc_at(q_desc0, (slot<2>(n) * TILES + i) * (Q4_BYTES / 16)), k_desc, sfk_desc, &sm.s_full[i][slot<2>(g)]);
        }
        f4_copies_sync();
        if (++t == k_tiles) t = 0, ++n;
    }
#pragma unroll
    for (int i = 0; i < TILES; ++i) f4_s_free_sync(i);
    commit_elected(&sm.drain[0]);  // whatever was issued must finish before tensor memory is freed
    mbar_wait_line(&sm.drain[0], 0, &sm.alone[0], nullptr, 0);
    __syncwarp();
}

// All copies.  The scores warp meets this one when it has issued S(g), and that says what is free, so that no copy has to wait
// for anything:
//   K4(g + 3) takes the slot of K4(g - 1), whose scores both query tiles have taken
//   V4(g + 3) (with the smoothing term) takes the slot of V4(g - 5): the softmax that took the scores of g - 1 had before, at
//             g - 3, waited for P.V(g - 5)
//   Q4 of the item after the next, at an item's first key tile: every score of the item before has been taken
static_assert(F4_K_RING == 4 && F4_V_RING == 8, "see above");
template <int TILES>
__device__ __forceinline__ void f4_copy_warp(Fp4Smem<TILES>& sm, const Fp4Args& a, int k_tiles) {
    const int n_items = a.items.mine(), total = n_items * k_tiles;
    auto item_of = [&](int n) { return int(blockIdx.x) + n * int(gridDim.x); };
    auto copy_q = [&](int n) {
        const int item = item_of(n);
        const size_t first = size_t(a.items.head(item)) * a.items.allocated + TILES * a.items.tile(item);
        if (elect_one()) {
            uint64_t* full = &sm.q_full[slot<2>(n)];
            mbar_expect_tx(full, TILES * (Q4_BYTES + SFQ_BYTES));
            bulk_load(sm.q[slot<2>(n)], a.q4 + first * Q4_BYTES, TILES * Q4_BYTES, full);
            bulk_load(sm.sfq[slot<2>(n)], a.sfq + first * (SFQ_BYTES / 4), TILES * SFQ_BYTES, full);
        }
        __syncwarp();
    };
    // where the next K4 and V4 tiles to be copied are: the block's item, the key tile in it, the tile in memory
    int ck = 0, nk = 0, tk = 0, cv = 0, nv = 0, tv = 0;
    size_t tile_k = size_t(a.items.head(item_of(0))) * k_tiles, tile_v = tile_k;
    const float* bias_row = nullptr;
    auto bias_of = [&](int n) {
        const int item = item_of(n);
        return a.bias + (size_t(a.items.head(item)) * a.q_blocks + (TILES * QUERY_TILE * a.items.tile(item)) / a.smooth_q) * (size_t(k_tiles) * KEY_TILE);
    };
    if (a.bias) bias_row = bias_of(0);
    auto copy_k = [&]() {
        if (ck >= total) return;
        if (elect_one()) {
            uint64_t* full = &sm.k_full[slot<F4_K_RING>(ck)];
            mbar_expect_tx(full, K4_BYTES + SFK_BYTES);
            bulk_load(sm.k[slot<F4_K_RING>(ck)], a.k4 + tile_k * K4_BYTES, K4_BYTES, full);
            bulk_load(sm.sfk[slot<F4_K_RING>(ck)], a.sfk + tile_k * (SFK_BYTES / 4), SFK_BYTES, full);
        }
        __syncwarp();
        ++ck, ++tile_k;
        if (++tk == k_tiles && ++nk < n_items) tk = 0, tile_k = size_t(a.items.head(item_of(nk))) * k_tiles;
    };
    auto copy_v = [&]() {
        if (cv >= total) return;
        if (elect_one()) {
            uint64_t* full = &sm.v_full[slot<F4_V_RING>(cv)];
            mbar_expect_tx(full, V4_BYTES + SFV_BYTES + (bias_row ? BIAS_BYTES : 0));
            bulk_load(sm.v[slot<F4_V_RING>(cv)], a.v4 + tile_v * V4_BYTES, V4_BYTES, full);
            bulk_load(sm.sfv[slot<F4_V_RING>(cv)], a.sfv + tile_v * (SFV_BYTES / 4), SFV_BYTES, full);
            if (bias_row) bulk_load(sm.bias[slot<F4_V_RING>(cv)], bias_row + size_t(tv) * KEY_TILE, BIAS_BYTES, full);
        }
        __syncwarp();
        ++cv, ++tile_v;
        if (++tv == k_tiles && ++nv < n_items) {
            tv = 0, tile_v = size_t(a.items.head(item_of(nv))) * k_tiles;
            if (a.bias) bias_row = bias_of(nv);
        }
    };
    copy_q(0);
    for (int i = 0; i < F4_K_RING; ++i) copy_k(), copy_v();
    for (int i = F4_K_RING; i < F4_V_RING; ++i) copy_v();
    if (n_items > 1) copy_q(1);
    int n = 0, t = 0;
#pragma unroll 1
    for (int g = 0; g < total; ++g) {
        f4_copies_sync();
        if (g >= 1) copy_k();
        if (g >= 5) copy_v();
        if (t == 0 && n >= 1 && n + 1 < n_items) copy_q(n + 1);
        if (++t == k_tiles) t = 0, ++n;
    }
    // After a wait that gave up, copies may still be in flight: the block's shared memory must not go away under them.  (Should
    // the first of these waits give up too, the others have been in flight all the while.)
    if (__any_sync(0xffffffffu, *static_cast<volatile int*>(&sm.abort_flag))) {
        for (int i = max(0, total - F4_V_RING); i < total; ++i) mbar_wait_line(&sm.v_full[slot<F4_V_RING>(i)], round_parity<F4_V_RING>(i), &sm.alone[1], nullptr, 0);
        for (int i = max(0, total - F4_K_RING); i < total; ++i) mbar_wait_line(&sm.k_full[slot<F4_K_RING>(i)], round_parity<F4_K_RING>(i), &sm.alone[1], nullptr, 0);
        for (int i = max(0, n_items - 2); i < n_items; ++i) mbar_wait_line(&sm.q_full[slot<2>(i)], round_parity<2>(i), &sm.alone[1], nullptr, 0);
    }
    __syncwarp();
}

// P.V(g) of query tile i as soon as P4(g) is delivered and V4(g) is there (and, at an item's first key tile, the O of the item
// before has been read).
template <int TILES>
__device__ __forceinline__ void f4_pv_warp(Fp4Smem<TILES>& sm, const Fp4Args& a, int k_tiles, uint32_t tmem, int i) {
    const int total = a.items.mine() * k_tiles;
    const uint32_t base = tmem + 256 * i;
    const uint64_t p_desc0 = smem_desc(smem_u32(sm.p[i][0]), QUERY_TILE * 16, 128), v_desc0 = smem_desc(smem_u32(sm.v[0]), V4_TILE_ROWS * 16, 128);
    const uint64_t sfp_desc0 = smem_desc(smem_u32(sm.sfp[i][0]), 16, 128), sfv_desc0 = smem_desc(smem_u32(sm.sfv[0]), 16, 128);
    int t = 0;
#pragma unroll 1
    for (int g = 0; g < total; ++g) {
        mbar_wait_line(&sm.v_full[slot<F4_V_RING>(g)], round_parity<F4_V_RING>(g), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        if (t == 0 && g > 0) f4_o_read_sync(i);
        f4_pv_sync(i, slot<2>(g));
        tc_fence_after();
        f4_issue_pv(base, desc_at(p_desc0, slot<2>(g) * (P4_BYTES / 16)), desc_at(v_desc0, slot<F4_V_RING>(g) * (V4_BYTES / 16)),
                    desc_at(sfp_desc0, slot<2>(g) * 32), desc_at(sfv_desc0, slot<F4_V_RING>(g) * (SFV_BYTES / 16)), t > 0, &sm.pv_done[i][slot<2>(g)]);
        if (++t == k_tiles) t = 0;
    }
    commit_elected(&sm.drain[1 + i]);
    mbar_wait_line(&sm.drain[1 + i], 0, &sm.alone[2 + i], nullptr, 0);
    __syncwarp();
}

// ---------------------------------------------------------------------------------------------------------------------
// softmax: query tile `qt`, key tiles g = w, w + 2, ..; thread = query row

template <int TILES, bool CODES>
__device__ __forceinline__ void f4_softmax(Fp4Smem<TILES>& sm, const Fp4Args& a, int k_tiles, uint32_t tmem, int qt, int w, int quarter, int lane) {
    const int row = quarter * 32 + lane, n_items = a.items.mine(), total = n_items * k_tiles;
    const uint32_t my = tmem + (uint32_t(quarter * 32) << 16) + qt * 256;
    const bool smoothed = a.bias != nullptr;
    int n = w / k_tiles, t = w % k_tiles;  // the block's item and the key tile in it
    auto item_of = [&](int i) { return int(blockIdx.x) + i * int(gridDim.x); };
    auto factor_of = [&](int i) {  // scores to the log2 domain
        const int h = a.items.head(item_of(i));
        return (a.k_outer ? fmaxf(a.qk_outer[h] * a.k_outer[h], 1e-30f) : a.qk_outer[h]) * a.scale_log2;
    };
    bool ok = true;
    float c = w < total ? factor_of(n) : 0.0f;
#pragma unroll 1
    for (int g = w; g < total; g += 2) {
        // the scores, and V's tile, with which the smoothing term arrives (usually long ago)
        const int stage = slot<F4_V_RING>(g);
        const bool there = mbar_try(&sm.v_full[stage], round_parity<F4_V_RING>(g));
        ok &= mbar_wait_line(&sm.s_full[qt][w], (g >> 1) & 1, &sm.abort_flag, a.status, STATUS_WAIT_SCORES);
        if (!there) ok &= mbar_wait_line(&sm.v_full[stage], round_parity<F4_V_RING>(g), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        __syncwarp();
        tc_fence_after();
        float2 x[KEY_TILE / 2];
        tmem_ld64_sync(my + F4_S, x);
        tc_fence_before();
        f4_s_free_arrive(qt);  // the scores are in registers
        // Scores in the log2 domain plus the smoothing term (or zeros); -inf in the slots past the last key, which keeps them
        // out of the maxima and makes their P zero.
        {
            const float2 c2 = make_float2(c, c);
            const float4* b4 = reinterpret_cast<const float4*>(smoothed ? sm.bias[stage] : sm.mask[(t + 1) * KEY_TILE > a.n_keys]);
#pragma unroll
            for (int j = 0; j < KEY_TILE / 4; ++j) {
                const float4 b = b4[j];
                x[2 * j] = fma2(x[2 * j], c2, make_float2(b.x, b.y));
                x[2 * j + 1] = fma2(x[2 * j + 1], c2, make_float2(b.z, b.w));
            }
        }
        float block_max[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            float top = fmaxf(x[8 * b].x, x[8 * b].y);
#pragma unroll
            for (int i = 1; i < 8; ++i) top = max3(top, x[8 * b + i].x, x[8 * b + i].y);
            block_max[b] = top;
        }
        const float tile_max = fmaxf(fmaxf(block_max[0], block_max[1]), fmaxf(block_max[2], block_max[3]));
        // the running maximum of the tile before, from the other warpgroup, and on to it
        if (g > 0) f4_max_sync(qt, w);
        const float before = t == 0 ? -INFINITY : sm.m[qt][w ^ 1][row];
        const float m = fmaxf(before, tile_max);
        sm.m[qt][w][row] = m;
        if (g + 1 < total) f4_max_arrive(qt, w ^ 1);
        // P.V(g - 2) has read this warpgroup's P^: asked now, looked at after the exponentials
        const int turn = g >> 1;
        const bool p_free = g < 2 || mbar_try(&sm.pv_done[qt][w], (turn - 1) & 1);

        // P in NVFP4: per 16 slots a scale byte sp = e4m3(max P / 6) with P = 1024 * 2^(x - m), then the codes of
        // P / sp = 2^(x - m + 10 - log2 sp) straight out of the exponent unit; log2 of every e4m3 value comes from a
        // table (a logarithm here would double the block's dependent chain).
        uint32_t codes[8], sf_word = 0;
        const float gain = P_LOG2_GAIN - m;
        float2 shift2[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float top = ex2(block_max[b] + gain) * (1.0f / 6.0f);
            const uint32_t byte = __nv_cvt_float_to_fp8(top, __NV_SATFINITE, __NV_E4M3);
            const float shift = gain - sm.log2_e4m3[byte];  // byte 0 (every P below e4m3's range): -inf, all codes zero
            shift2[b] = make_float2(shift, shift);
            sf_word |= byte << (8 * b);
        }
        const float alpha = ex2(before - m);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float2 r[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 e = add2(x[8 * b + 4 * half + i], shift2[b]);
                    r[i] = make_float2(ex2(e.x), ex2(e.y));
                }
                codes[2 * b + half] = e2m1x8(r);
            }
        }
        auto first_row = [&]() { return (TILES * a.items.tile(item_of(n)) + qt) * QUERY_TILE + quarter * 32; };  // of this warp
        if (CODES && first_row() + lane < a.n_queries) {  // diagnostics: this row's P^ of the tile, 8 words of codes and the 4 scale bytes
            uint32_t* dst = a.p_words + ((size_t(a.items.head(item_of(n))) * a.n_queries + first_row() + lane) * k_tiles + t) * 9;
#pragma unroll
            for (int i = 0; i < 8; ++i) dst[i] = codes[i];
            dst[8] = sf_word;
        }
        if (!p_free) ok &= mbar_wait_line(&sm.pv_done[qt][w], (turn - 1) & 1, &sm.abort_flag, a.status, STATUS_WAIT_PV);
        *reinterpret_cast<uint4*>(sm.p[qt][w] + row * 16) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
        *reinterpret_cast<uint4*>(sm.p[qt][w] + QUERY_TILE * 16 + row * 16) = make_uint4(codes[4], codes[5], codes[6], codes[7]);
        sm.sfp[qt][w][lane][quarter] = sf_word;  // byte 2 piece + block
        // Where a row's maximum moved, O and the denominator shrink by alpha once P.V(g - 1) is done.
        if (t > 0 && !__all_sync(0xffffffffu, alpha == 1.0f)) {
            ok &= mbar_wait_line(&sm.pv_done[qt][w ^ 1], ((g - 1) >> 1) & 1, &sm.abort_flag, a.status, STATUS_WAIT_PV);
            __syncwarp();
            tc_fence_after();
            const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll
            for (int first = 0; first < HEAD_DIM; first += 64) {  // 128 channels, then the denominator's column (the 15 after it stay zero)
                float2 o[4][8];
#pragma unroll
                for (int i = 0; i < 4; ++i) tmem_ld16_async(my + F4_O + first + 16 * i, o[i]);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    reg_fence8(o[i]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[i][j] = mul2(o[i][j], alpha2);
                    tmem_st16(my + F4_O + first + 16 * i, o[i]);
                }
            }
            float2 sum[4];
            tmem_ld8_async(my + F4_O + HEAD_DIM, sum);
            tmem_wait_ld();
            reg_fence4(sum);
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j] = mul2(sum[j], alpha2);
            tmem_st8(my + F4_O + HEAD_DIM, sum);
            tmem_wait_st();
        }
        tc_fence_before();
        fence_proxy_async();  // P^ and its scale bytes are read by the tensor pipe (tcgen05.cp, tcgen05.mma)
        __syncwarp();
        f4_pv_arrive(qt, w);

        if (t + 1 == k_tiles) {  // the item is done: its rows out
            ok &= mbar_wait_line(&sm.pv_done[qt][w], turn & 1, &sm.abort_flag, a.status, STATUS_WAIT_PV);
            ok = __all_sync(0xffffffffu, ok && !gave_up(sm.abort_flag));
            tc_fence_after();
            if (n > 0 && ((g - k_tiles) & 1) != w) f4_staged_sync(qt);  // the item before was stored by the other warpgroup
            bulk_store_read_wait();
            const int head = a.items.head(item_of(n));
            const float4* scale4 = reinterpret_cast<const float4*>(a.v_outer + size_t(head) * HEAD_DIM);
            float2 last[4];
            tmem_ld8_async(my + F4_O + HEAD_DIM, last);  // column 128: the sum of P^
            tmem_wait_ld();
            reg_fence4(last);
            const float inv = 1.0f / last[0].x;
            uint8_t* staged = sm.staged[qt][quarter];
#pragma unroll
            for (int part = 0; part < HEAD_DIM / 16; ++part) {
                float2 o[8];
                tmem_ld16_sync(my + F4_O + part * 16, o);
                uint32_t word[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 s = scale4[part * 4 + i];
                    word[2 * i] = output_pair(o[2 * i].x * s.x * inv, o[2 * i].y * s.y * inv, a.out_layout.half);
                    word[2 * i + 1] = output_pair(o[2 * i + 1].x * s.z * inv, o[2 * i + 1].y * s.w * inv, a.out_layout.half);
                }
                *reinterpret_cast<uint4*>(staged + lane * STAGED_PITCH + part * 32) = make_uint4(word[0], word[1], word[2], word[3]);
                *reinterpret_cast<uint4*>(staged + lane * STAGED_PITCH + part * 32 + 16) = make_uint4(word[4], word[5], word[6], word[7]);
            }
            tc_fence_before();
            if (g + 1 < total) f4_o_read_arrive(qt);
            send_staged_rows(staged, lane, first_row(), a.n_queries, head, a.out, a.out_layout, a.peers, ok);
            if (n + 1 < n_items && ((g + k_tiles) & 1) != w) {
                bulk_store_read_wait();
                __syncwarp();
                f4_staged_arrive(qt);
            }
        }
        if ((t += 2) >= k_tiles) {
            for (; t >= k_tiles; t -= k_tiles) ++n;
            if (g + 2 < total) c = factor_of(n);
        }
    }
    bulk_store_read_wait();
}

template <int TILES, bool CODES>
__global__ void __launch_bounds__(F4_THREADS<TILES>, 1) attention_fp4_kernel(const __grid_constant__ Fp4Args a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    Fp4Smem<TILES>& sm = *reinterpret_cast<Fp4Smem<TILES>*>(smem_raw);
    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x / 32), 0), lane = threadIdx.x % 32;  // (the shuffle tells the compiler that it is uniform)
    const int k_tiles = (a.n_keys + KEY_TILE - 1) / KEY_TILE;

    if (threadIdx.x == 0) {
        sm.abort_flag = 0;
        for (int& word : sm.alone) word = 0;
        for (int s = 0; s < 2; ++s) mbar_init(&sm.q_full[s], 1);
        for (int s = 0; s < F4_K_RING; ++s) mbar_init(&sm.k_full[s], 1);
        for (int s = 0; s < F4_V_RING; ++s) mbar_init(&sm.v_full[s], 1);
        for (int i = 0; i < TILES; ++i)
            for (int w = 0; w < 2; ++w) mbar_init(&sm.s_full[i][w], 1), mbar_init(&sm.pv_done[i][w], 1);
        for (int i = 0; i < 1 + TILES; ++i) mbar_init(&sm.drain[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x >= 128 && threadIdx.x < 256) {
        const int byte = threadIdx.x - 128;
        const float value = __half2float(__half(__nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte), __NV_E4M3)));
        sm.log2_e4m3[byte] = value > 0.0f ? log2f(value) : INFINITY;  // byte 127 is NaN: never produced (satfinite)
    }
    if (threadIdx.x >= 256 && threadIdx.x < 256 + KEY_TILE) {
        const int at = threadIdx.x - 256, j = at % F4_HALF_SLOTS;
        const int key = (k_tiles - 1) * KEY_TILE + F4_HALF_SLOTS * (at / F4_HALF_SLOTS) + 8 * (j % 8 / 2) + 2 * (j / 8) + j % 2;  // slot -> key
        sm.mask[0][at] = 0.0f;
        sm.mask[1][at] = key < a.n_keys ? 0.0f : -INFINITY;
    }
    if (warp == 0) tmem_alloc(&sm.tmem_base, 256 * TILES);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);
    wait_for_previous_kernel();

    if (warp >= F4_SOFTMAX_WARP) {
        if constexpr (TILES == 2) set_registers<F4_SOFTMAX_REGISTERS, F4_LAUNCH_REGISTERS>();
        const int group = (warp - F4_SOFTMAX_WARP) / 4;
        f4_softmax<TILES, CODES>(own_view(sm), a, k_tiles, tmem, group >> 1, group & 1, warp % 4, lane);
    } else {
        if constexpr (TILES == 2) set_registers<F4_SERVICE_REGISTERS, F4_LAUNCH_REGISTERS>();
        if (warp == F4_SCORES_WARP)
            f4_scores_warp(own_view(sm), a, k_tiles, tmem);
        else if (warp == F4_COPY_WARP)
            f4_copy_warp(own_view(sm), a, k_tiles);
        else if (warp < F4_PV_WARP + TILES)
            f4_pv_warp(own_view(sm), a, k_tiles, tmem, warp - F4_PV_WARP);
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(sm.tmem_base, 256 * TILES);
    }
}

}  // namespace unica

using namespace unica;

static constexpr int F4_MAX_DEVICES = 64;

// One query tile per block where that takes less time: a block takes two thirds of the time of a pair's for a key tile (1 head x 8192 tokens
// 126.0 -> 82.4 us, 4 x 1024 24.4 -> 17.9, 18 x 1024 25.1 -> 19.2; 16 x 1000 queries, 77 keys 9.6 -> 9.0), so it depends on the rounds that
// the blocks of either kind go.  Their results are the same.
extern "C" int unica_b200_fast_item_rows(int heads, int n_queries, int sms) {
    if (heads <= 0 || n_queries <= 0 || sms <= 0) return 0;
    const auto rounds = [&](int rows) { return ((n_queries + rows - 1LL) / rows * heads + sms - 1) / sms; };
    return 2 * rounds(QUERY_TILE) < 3 * rounds(2 * QUERY_TILE) ? QUERY_TILE : 2 * QUERY_TILE;
}

int unica_attention_fp4(const uint8_t* q4, const void* sfq, const uint8_t* k4, const void* sfk, const uint8_t* v4, const void* sfv,
                         const float* qk_outer, const float* k_outer, const float* v_outer, const float* bias, int q_blocks, int smooth_q, void* out,
                         void* const* peer_out, int n_peers, unica_token_layout out_layout, int heads, int n_queries, int n_keys,
                         float scale_log2, uint32_t* p_words, int* status, void* stream, bool overlapped) {
    if (!q4 || !sfq || !k4 || !sfk || !v4 || !sfv || !qk_outer || !v_outer || !out) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_fp4: null pointer");
    if (heads <= 0 || heads > 65535 || n_queries <= 0 || n_keys <= 0)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_fp4: heads must be in 1..65535, n_queries and n_keys positive");
    if (bias && (smooth_q <= 0 || smooth_q % 256 || q_blocks != (n_queries + smooth_q - 1) / smooth_q))
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_fp4: with a smoothing term, smooth_q must be a multiple of 256 and q_blocks = ceil(n_queries / smooth_q)");
    PeerOutputs peers = {};
    if (int e = unica_peer_outputs(out, peer_out, n_peers, &peers)) return e;
    if (int e = unica_check_device()) return e;
    Fp4Args args = {};
    args.q4 = q4, args.k4 = k4, args.v4 = v4;
    args.sfq = static_cast<const uint32_t*>(sfq), args.sfk = static_cast<const uint32_t*>(sfk), args.sfv = static_cast<const uint32_t*>(sfv);
    args.qk_outer = qk_outer, args.k_outer = k_outer, args.v_outer = v_outer, args.bias = bias, args.q_blocks = q_blocks, args.smooth_q = smooth_q > 0 ? smooth_q : 1;
    args.out = static_cast<__nv_bfloat16*>(out), args.out_layout = to_layout(out_layout), args.peers = peers;
    args.n_queries = n_queries, args.n_keys = n_keys, args.scale_log2 = scale_log2, args.p_words = p_words, args.status = status;
    const long long pairs = (n_queries + 2 * QUERY_TILE - 1) / (2 * QUERY_TILE), tiles = (n_queries + QUERY_TILE - 1) / QUERY_TILE;  // Q4 holds an even number of tiles
    if (pairs * heads > INT_MAX / 2) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_fp4: more than 2^30 pairs of query tiles");
    int sms = 0;  // persistent blocks, one per SM
    if (int e = unica_sm_count(&sms)) return e;
    auto launch = [&](auto kernel, int threads, int smem, int instance) -> int {
        // Set up once per kernel instance and device, as in attention_int8.cu.
        static std::atomic<bool> ready[3][F4_MAX_DEVICES];
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess) return unica_check_launch("attention_fp4 (device)");
        if (device >= F4_MAX_DEVICES || !ready[instance][device].load(std::memory_order_acquire)) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
                cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess)
                return unica_check_launch("attention_fp4 (shared memory size)");
            cudaFuncAttributes attributes;
            if (cudaFuncGetAttributes(&attributes, kernel) != cudaSuccess) return unica_check_launch("attention_fp4 (attributes)");
            if (threads == F4_THREADS<2> && attributes.numRegs * threads < F4_SPLIT_REGISTERS)
                return unica_fail(UNICA_B200_ERR_KERNEL, "attention_fp4: this build holds fewer registers per block than its setmaxnreg split needs");
            if (device < F4_MAX_DEVICES) ready[instance][device].store(true, std::memory_order_release);
        }
        launch_after(kernel, dim3(args.items.count < sms ? args.items.count : sms), threads, size_t(smem), static_cast<cudaStream_t>(stream), overlapped, args);
        return unica_check_launch("attention_fp4");
    };
    const bool single = !p_words && unica_b200_fast_item_rows(heads, n_queries, sms) == QUERY_TILE;
    args.items.tiles = int(single ? tiles : pairs), args.items.allocated = int(2 * pairs), args.items.count = args.items.tiles * heads;
    return single    ? launch(attention_fp4_kernel<1, false>, F4_THREADS<1>, int(sizeof(Fp4Smem<1>)) + 128, 2)
           : p_words ? launch(attention_fp4_kernel<2, true>, F4_THREADS<2>, int(sizeof(Fp4Smem<2>)) + 128, 1)
                     : launch(attention_fp4_kernel<2, false>, F4_THREADS<2>, int(sizeof(Fp4Smem<2>)) + 128, 0);
}

extern "C" int unica_b200_attention_fp4(const uint8_t* q4, const void* sfq, const uint8_t* k4, const void* sfk, const uint8_t* v4,
                                        const void* sfv, const float* qk_outer, const float* v_outer, const float* bias,
                                        int q_blocks, int smooth_q, void* out, unica_token_layout out_layout, int heads,
                                        int n_queries, int n_keys, float scale_log2, int* status, void* stream) {
    return unica_attention_fp4(q4, sfq, k4, sfk, v4, sfv, qk_outer, nullptr, v_outer, bias, q_blocks, smooth_q, out, nullptr, 0, out_layout, heads,
                         n_queries, n_keys, scale_log2, nullptr, status, stream);
}

extern "C" int unica_b200_attention_fp4_peers(const uint8_t* q4, const void* sfq, const uint8_t* k4, const void* sfk,
                                              const uint8_t* v4, const void* sfv, const float* qk_outer, const float* v_outer,
                                              const float* bias, int q_blocks, int smooth_q, void* out, void* const* peer_out,
                                              int n_peers, unica_token_layout out_layout, int heads, int n_queries, int n_keys,
                                              float scale_log2, int* status, void* stream) {
    return unica_attention_fp4(q4, sfq, k4, sfk, v4, sfv, qk_outer, nullptr, v_outer, bias, q_blocks, smooth_q, out, peer_out, n_peers, out_layout, heads,
                         n_queries, n_keys, scale_log2, nullptr, status, stream);
}

extern "C" int unica_b200_attention_fp4_codes(const uint8_t* q4, const void* sfq, const uint8_t* k4, const void* sfk,
                                              const uint8_t* v4, const void* sfv, const float* qk_outer, const float* v_outer,
                                              const float* bias, int q_blocks, int smooth_q, void* out, unica_token_layout out_layout,
                                              int heads, int n_queries, int n_keys, float scale_log2, uint32_t* p_words, int* status,
                                              void* stream) {
    if (!p_words) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_fp4_codes: null pointer");
    return unica_attention_fp4(q4, sfq, k4, sfk, v4, sfv, qk_outer, nullptr, v_outer, bias, q_blocks, smooth_q, out, nullptr, 0, out_layout, heads,
                         n_queries, n_keys, scale_log2, p_words, status, stream);
}

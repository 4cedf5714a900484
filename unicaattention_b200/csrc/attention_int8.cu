// The accurate mode's flash-attention loop on tcgen05 (replaces the reference's attention_int8pv_tma, csrc/flash.cu:806-959).
//
// Persistent blocks, one of 16 warps per SM, each taking tiles of 128 query rows (items) blockIdx.x, blockIdx.x +
// gridDim.x, ...  Four warpgroups with three kinds of work (a thread of a computing warpgroup owns one query row = one
// tensor-memory lane, so row maxima and sums need no shuffles):
//
//   softmax A, B   every other key tile each: the scores S(g) of tensor memory, read once into registers, become the bytes
//                  P^(g) = rint(255 * 2^(x - tile max)) of the A-operand image in shared memory; the tile maximum and the
//                  row sum go to the flush threads through shared memory.  They carry nothing from tile to tile.
//   flush          out = out * alpha + beta * float(acc(g)) for every key tile g, the row's 128 outputs in registers;
//                  they own the running exponent and the denominator, and write the result.
//   service        two warps: the scores' instructions and all bulk TMA copies (contiguous 8 KB images written by the
//                  quantizers, K8 and V8 in rings of their own), and P.V's instructions:
//
//   S(g)   = Q8 . K8(g)^T      kind::i8 s8 x s8 -> s32, 128 x 64, 4 instructions of K = 32, a ring of 4 buffers
//   acc(g) = P^(g) . V8(g)     kind::i8 u8 x u8 -> s32, 128 x 128, 2 instructions of K = 32, two accumulators (g even / odd);
//                              V8 is stored as 128 plus or minus its codes, see flush32
//
// (The copies are in the scores warp because a warp of their own, meeting it once per tile, measured 7 % slower.)
//
// Key tiles are counted across items (g), and every ring runs on from one item to the next: while the flush warps normalise
// and store an item, the copies, scores and exponentials of the next one are under way.  With one block per item a block's
// start (5500 cycles to the first P.V) and end (11700) were exposed, a fifth of a call of 4128 tokens.
//
// What bounds it: issue slots.  A key tile costs a scheduler some 590 instructions, of which 145 packed FP32 ones count twice
// (an fma.f32x2 issues for two cycles), and the three computing warps of a scheduler keep it about 76 % busy: 967 cycles
// per tile.  The tensor pipe is active 256 cycles of a tile (320 with its shared-memory reads), the exponential unit 512.
// Hence:
//   - nothing waits in a loop where it can be helped: hand-overs between warps are named barriers, on which the hardware
//     blocks a warp (probing loops had grown to half of all issued instructions), and the copies are issued where their
//     slots are known to be free, so that nobody polls for them;
//   - the accumulators are added up without a conversion to float (flush32), and P^ is rounded without one (softmax_tile);
//   - the flush warps load the next accumulator while they add up the present one, the softmax warps ask for their next scores
//     while the exponentials run: a probe's answer takes some sixty cycles.
//
// Numerics (bench/emulate.py:298-369 with the accurate contract): scores in the log2 domain, c = (q_scale * k_scale) *
// log2(e) / sqrt(d); P^ as u8 against the tile's own maximum; the denominator sums the rounded P^ (per channel) or
// p / s_j in float before rounding (per token); every tile is flushed as out = out * alpha + beta * acc with
// beta = 2^(m_tile - m) and alpha = 2^(m_old - m_new), where m is a reference exponent that follows the running maximum
// only in large steps (the common factor cancels against the denominator's).  The 255 stays in numerator and
// denominator alike (as csrc/flash.cu:409-414 does).
//
// Tensor memory (all 512 columns): S ring 4 x 64 | acc 2 x 128.  All waits are bounded (common.cuh).
#include <atomic>
#include <climits>

#include "attention_common.cuh"
#include "capi.h"

namespace unica {

// Warps 2 and 3 do nothing: registers are dealt out to whole warpgroups.
constexpr int SCORES_WARP = 0, PV_WARP = 1, FLUSH_WARP = 4, SOFTMAX_WARP = 8, ATT_WARPS = 16, ATT_THREADS = ATT_WARPS * 32;
// registers per thread after setmaxnreg; the block is launched with ATT_THREADS x LAUNCH_REGISTERS = 65536
constexpr int LAUNCH_REGISTERS = 128, SOFTMAX_REGISTERS = 120, FLUSH_REGISTERS = 232, SERVICE_REGISTERS = 40;
static_assert(128 * (2 * SOFTMAX_REGISTERS + FLUSH_REGISTERS + SERVICE_REGISTERS) <= ATT_THREADS * LAUNCH_REGISTERS, "the split must fit the launch");
constexpr int K_RING = 6;   // K8 tiles in shared memory: tile g + K_RING - S_RING is fetched when S(g) is issued (see scores_warp)
constexpr int V_RING = 8;   // V8 tiles (and the keys' scales, per token): tile g - V_LATER is fetched when S(g) is issued
constexpr int S_RING = 4;   // score buffers in tensor memory
constexpr int P_RING = 4;   // P^ images in shared memory
constexpr int ST_RING = 8;  // (tile maximum, row sum) records on their way from the softmax to the flush threads
// The record of tile g is overwritten by the softmax of tile g + ST_RING, which waits for the flush of tile g + ST_RING - P_RING.
static_assert(ST_RING > P_RING, "a record must have been read before it is overwritten");
constexpr int Q_BYTES = QUERY_TILE * HEAD_DIM;  // 16384
constexpr int K_BYTES = KEY_TILE * HEAD_DIM;    // 8192
constexpr int V_BYTES = KEY_TILE * HEAD_DIM;    // 8192
constexpr int TOK_BYTES = 2 * KEY_TILE * 4;     // 512
constexpr int P_BYTES = QUERY_TILE * KEY_TILE;  // 8192
constexpr int SCALE_BYTES = HEAD_DIM * 4;       // 512
constexpr int TMEM_COLUMNS = 512;
constexpr int COL_S = 0, COL_ACC = 256;
constexpr int OUTLIER_BATCH = 16;  // outlier keys whose rows are in shared memory at a time (the epilogue of the outliers mode)
constexpr float P_UNIT = 1.40129846432481707e-45f;  // 2^-149, see softmax_tile
constexpr float REFERENCE_SLACK = 60.0f;  // log2: how far a tile maximum may rise above a row's reference exponent

struct __align__(128) AttSmem {
    int8_t q[2][Q_BYTES];
    int8_t k[K_RING][K_BYTES];
    int8_t v[V_RING][V_BYTES];
    uint8_t p[P_RING][P_BYTES];
    uint8_t staged[4][32 * STAGED_PITCH];
    float2 st[ST_RING][QUERY_TILE];
    uint16_t p_sum[ST_RING][QUERY_TILE];  // per token: sum of the row's P^ (per channel it is the record's own sum)
    float v_scale[2][HEAD_DIM];
    float tok[V_RING][2 * KEY_TILE];
    uint64_t q_full[2], q_free[2], k_full[K_RING], v_full[V_RING], s_full[S_RING], acc_full[2], drain[2];
    uint32_t tmem_base;
    int abort_flag;
    int alone[2];  // zeros: a word for each warp that drains what it issued, which no other warp's wait may cut short
};
static_assert(sizeof(AttSmem) + 128 <= 227 * 1024, "the block's shared memory");

// Hand-overs between warps are named barriers: the receiving warp is blocked by the hardware, at no cost in issue slots, and
// runs again some 40 cycles after the last arrival (an mbarrier: 115).  A wait on an mbarrier is a loop of probes, whose
// instructions the computing warps of the same scheduler pay for: with mbarriers everywhere, half of all issued instructions
// were waiting loops.  What the copies and the tensor core complete can only be waited for on an mbarrier.
constexpr int BAR_FLUSH = 1, BAR_S_FREE = 2, BAR_PV = BAR_S_FREE + S_RING, BAR_P_FREE = BAR_PV + P_RING;
static_assert(BAR_P_FREE + P_RING <= 16, "a block has sixteen named barriers");
// scores buffer: the four softmax warps of its tile, to the scores warp
__device__ __forceinline__ void s_free_arrive(int g) { asm volatile("bar.arrive %0, 160;" ::"r"(BAR_S_FREE + slot<S_RING>(g)) : "memory"); }
__device__ __forceinline__ void s_free_sync(int g) { asm volatile("bar.sync %0, 160;" ::"r"(BAR_S_FREE + slot<S_RING>(g)) : "memory"); }
// what P.V(g) needs: P^(g) from the four softmax warps of tile g, and the accumulator from the four flush warps, which have
// read tile g - 2 out of it (for g < 2 they arrive before their first tile)
__device__ __forceinline__ void pv_arrive(int g) { asm volatile("bar.arrive %0, 288;" ::"r"(BAR_PV + slot<P_RING>(g)) : "memory"); }
// P^ image: the four flush warps, which have seen P.V(g) complete, to the four softmax warps that write P^(g + P_RING)
__device__ __forceinline__ void p_free_arrive(int g) { asm volatile("bar.arrive %0, 256;" ::"r"(BAR_P_FREE + slot<P_RING>(g)) : "memory"); }
__device__ __forceinline__ void p_free_sync(int g) { asm volatile("bar.sync %0, 256;" ::"r"(BAR_P_FREE + slot<P_RING>(g)) : "memory"); }
__device__ __forceinline__ void pv_sync(int g) { asm volatile("bar.sync %0, 288;" ::"r"(BAR_PV + slot<P_RING>(g)) : "memory"); }

constexpr uint32_t IDESC_QK = idesc_i8(true, QUERY_TILE, KEY_TILE);
constexpr uint32_t IDESC_PV = idesc_u8(QUERY_TILE, HEAD_DIM);

// 32 accumulator values into 32 of a row's sums.  The accumulators are sums of products of bytes (V8 is stored plus V8_BIAS, negated in odd tiles),
// integers in 0 .. 64 * 255 * 255 < 2^23, and the bits of such an integer are those of the denormal float integer * 2^-149: they
// go into the multiply-add as they are, where a conversion would cost an instruction per element.  The sums are kept times
// SUM_UNIT, so that the factor (beta times 2^149 times SUM_UNIT, beta up to 2^REFERENCE_SLACK) stays in range.
constexpr float BETA_UNIT = 9007199254740992.0f, SUM_UNIT = 1.2621774483536189e-29f;  // 2^53, 2^-96
static_assert(double(BETA_UNIT) * SUM_UNIT * (1ull << 43) == 1.0, "2^(149 - 96) and 2^-96");
// What the bias adds to a row's sums is known (V8_BIAS times the sum of its P^) and taken out every BIAS_TILES tiles.  With the sign
// alternating from tile to tile no more than about one tile's share of it is in them at a time: against sums in 64 bits they err by
// 5e-7 of their size after 65 tiles of plain values, and by 3.7e-6 with the shares of eight tiles in them.
constexpr int BIAS_TILES = 8;
__device__ __forceinline__ void flush32(const float2 (&y)[16], float2* o, float2 beta2) {
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = fma2(beta2, y[i], o[i]);
}

struct AttArgs {
    const int8_t *q8, *k8, *v8;
    const float *q_scale, *k_scale, *v_scale, *v_token;
    const int* outlier_keys;
    const float* outlier_rows;
    int n_outliers;
    __nv_bfloat16* out;
    TokenLayout out_layout;
    PeerOutputs peers;
    int n_queries, n_keys;
    Items items;
    float scale_log2;
    int* status;
};

// ---------------------------------------------------------------------------------------------------------------------
// the service warps; what they issue, one elected lane issues (see elect_one() in common.cuh)

// The tensor-core work of a tile in one statement, executed by a whole converged warp and issued by one elected lane: election
// and instructions under one predicate, with no branch around them.  `if (elect_one()) { .. }` inside a loop of the warp took
// twice the cycles on an idle SM (164 against 77 for P.V), and 550 between computing warps.
__device__ __forceinline__ void issue_scores(uint32_t d, uint64_t q_desc, uint64_t k_desc, uint64_t* full) {
    constexpr int Q_STEP = 2 * QUERY_TILE * 16 / 16, K_STEP = 2 * KEY_TILE * 16 / 16;
    asm volatile(
        "{\n\t"
        ".reg .pred e, acc;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "setp.eq.u32 acc, 0, 0;\n\t"  // the buffer holds MAGIC_BITS
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %9, acc;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %3, %4, %9, acc;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %5, %6, %9, acc;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %7, %8, %9, acc;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%10];\n\t"
        "}" ::"r"(d),
        "l"(q_desc), "l"(k_desc), "l"(desc_at(q_desc, Q_STEP)), "l"(desc_at(k_desc, K_STEP)), "l"(desc_at(q_desc, 2 * Q_STEP)), "l"(desc_at(k_desc, 2 * K_STEP)),
        "l"(desc_at(q_desc, 3 * Q_STEP)), "l"(desc_at(k_desc, 3 * K_STEP)), "r"(IDESC_QK), "r"(smem_u32(full))
        : "memory");
}
__device__ __forceinline__ void issue_pv(uint32_t d, uint64_t p_desc, uint64_t v_desc, uint64_t* full) {
    constexpr int P_STEP = 2 * QUERY_TILE * 16 / 16, V_STEP = 2 * HEAD_DIM * 16 / 16;
    asm volatile(
        "{\n\t"
        ".reg .pred e, first, acc;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "setp.ne.u32 first, 0, 0;\n\t"  // the first instruction of a tile overwrites the accumulator
        "setp.eq.u32 acc, 0, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %5, first;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %3, %4, %5, acc;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t"
        "}" ::"r"(d),
        "l"(p_desc), "l"(v_desc), "l"(desc_at(p_desc, P_STEP)), "l"(desc_at(v_desc, V_STEP)), "r"(IDESC_PV), "r"(smem_u32(full))
        : "memory");
    static_assert(KEY_TILE == 64 && HEAD_DIM == 128, "two instructions of K = 32 for P.V, four for the scores");
}

// S(g), as soon as K8(g) has landed and the softmax of tile g - S_RING has handed the scores buffer back; and all copies, none
// of which has to wait for anything:
//   K8(g + K_RING - S_RING)  (from g = S_RING on) takes the slot of K8(g - S_RING), whose scores have been read
//   V8(g - V_LATER)          takes the slot of V8(g - V_LATER - V_RING): the softmax of tile g - S_RING, which has just handed
//                            its buffer back, began after the flush of tile g - S_RING - P_RING had seen its P.V complete
//                            (p_free_sync).  Why later: this warp is busy for most of a tile's time, and P.V(g) is tiles away
//                            (copied with S(g), between its instructions and the copy of K8, 37 heads x 8192 tokens took 1.074
//                            ms per channel and 1.352 per token; so 1.066 and 1.329).  Why before the waits below: the flush
//                            leaves an item once the first P.V of the next is complete, so with k_tiles key tiles per head
//                            what frees Q8's slot for the item that starts with tile g is P.V(g - k_tiles).
//   Q8 of the item after the next, when V8's argument says that the flush has left the item before (Q_AHEAD tiles into the
//                            next; with fewer key tiles per head than that, when it is needed)
// The whole warp runs the loop and one elected lane issues.  A wait that gave up changes nothing here: instructions on
// whatever lies in the buffers do no harm (the result is not stored), and every hand-over still finds its receiver.
constexpr int V_LATER = 2, Q_AHEAD = V_RING + V_LATER;
static_assert(V_RING >= S_RING + P_RING, "see above");
template <bool V_TOKEN>
__device__ __forceinline__ void scores_warp(AttSmem& sm, const AttArgs& a, int k_tiles, uint32_t tmem) {
    const uint64_t q_desc0 = smem_desc(smem_u32(sm.q[0]), QUERY_TILE * 16, 128), k_desc0 = smem_desc(smem_u32(sm.k[0]), KEY_TILE * 16, 128);
    const int n_items = a.items.mine(), total = n_items * k_tiles;
    auto head_of = [&](int n) { return a.items.head(int(blockIdx.x) + n * int(gridDim.x)); };
    auto copy_q = [&](int n) {  // the block's nth item; its slot is free when the scores' instructions and the flush have left item n - 2
        mbar_wait_line(&sm.q_free[slot<2>(n)], round_parity<2>(n) ^ 1, &sm.abort_flag, a.status, STATUS_WAIT_STAGE);
        __syncwarp();
        const int item = int(blockIdx.x) + n * int(gridDim.x), head = a.items.head(item);
        if (elect_one()) {
            mbar_expect_tx(&sm.q_full[slot<2>(n)], Q_BYTES + SCALE_BYTES);
            bulk_load(sm.q[slot<2>(n)], a.q8 + (size_t(head) * a.items.allocated + a.items.tile(item)) * Q_BYTES, Q_BYTES, &sm.q_full[slot<2>(n)]);
            bulk_load(sm.v_scale[slot<2>(n)], a.v_scale + size_t(head) * HEAD_DIM, SCALE_BYTES, &sm.q_full[slot<2>(n)]);
        }
        __syncwarp();
    };
    // where K8's next tile is (its item, tile and head), and its slot; the same for V8's tile t of item n and the scores
    int nk = 0, tk = 0, k_slot = 0;
    const int8_t* k_src = a.k8 + size_t(head_of(0)) * k_tiles * K_BYTES;
    auto copy_k = [&]() {
        if (nk >= n_items) return;
        copy_elected(sm.k[k_slot], k_src, K_BYTES, &sm.k_full[k_slot]);
        k_src += K_BYTES;
        if (++k_slot == K_RING) k_slot = 0;
        if (++tk == k_tiles && ++nk < n_items) tk = 0, k_src = a.k8 + size_t(head_of(nk)) * k_tiles * K_BYTES;
    };
    copy_q(0);
    for (int i = 0; i < K_RING; ++i) copy_k();
    if (n_items > 1) copy_q(1);
    // V8's next tile
    const int v_later = k_tiles > 1 ? V_LATER : 1;
    int nv = 0, tv = 0, v_tile = 0;
    size_t tile = size_t(head_of(0)) * k_tiles;
    auto copy_v = [&]() {
        const int slot_v = slot<V_RING>(v_tile++);
        if (V_TOKEN) {
            if (elect_one()) {
                mbar_expect_tx(&sm.v_full[slot_v], V_BYTES + TOK_BYTES);
                bulk_load(sm.v[slot_v], a.v8 + tile * V_BYTES, V_BYTES, &sm.v_full[slot_v]);
                bulk_load(sm.tok[slot_v], a.v_token + tile * (2 * KEY_TILE), TOK_BYTES, &sm.v_full[slot_v]);
            }
            __syncwarp();
        } else {
            copy_elected(sm.v[slot_v], a.v8 + tile * V_BYTES, V_BYTES, &sm.v_full[slot_v]);
        }
        ++tile;
        if (++tv == k_tiles) tv = 0, tile = size_t(head_of(++nv)) * k_tiles;
    };
    int n = 0, t = 0, slot_k = 0, parity_k = 0;
#pragma unroll 1
    for (int g = 0; g < total; ++g) {
        s_free_sync(g);
        if (g >= v_later) copy_v();
        if (t == 0) {
            if (n >= 2 && k_tiles <= Q_AHEAD) copy_q(n);
            mbar_wait_line(&sm.q_full[slot<2>(n)], round_parity<2>(n), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        }
        mbar_wait_line(&sm.k_full[slot_k], parity_k, &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        __syncwarp();
        tc_fence_after();
        issue_scores(tmem + COL_S + slot<S_RING>(g) * KEY_TILE, desc_at(q_desc0, slot<2>(n) * (Q_BYTES / 16)), desc_at(k_desc0, slot_k * (K_BYTES / 16)),
                     &sm.s_full[slot<S_RING>(g)]);
        if (++slot_k == K_RING) slot_k = 0, parity_k ^= 1;
        if (g >= S_RING) copy_k();
        if (k_tiles > Q_AHEAD && t == Q_AHEAD && n >= 1 && n + 1 < n_items) copy_q(n + 1);
        if (++t == k_tiles) {
            commit_elected(&sm.q_free[slot<2>(n)]);
            t = 0, ++n;
        }
    }
    for (int b = 0; b < S_RING; ++b) {
        s_free_sync(total + b);  // every buffer has been handed back once more than it was used
        if (b < v_later && total + b >= v_later) copy_v();
    }
    commit_elected(&sm.drain[0]);  // whatever was issued must finish before tensor memory is freed
    mbar_wait_line(&sm.drain[0], 0, &sm.alone[0], nullptr, 0);
    // After a wait that gave up, copies may still be in flight: the block's shared memory must not go away under them.  (Should
    // the first of these waits give up too, the others have been in flight all the while.)
    if (__any_sync(0xffffffffu, *static_cast<volatile int*>(&sm.abort_flag))) {
        for (int i = max(0, total - V_RING); i < total; ++i) mbar_wait_line(&sm.v_full[slot<V_RING>(i)], round_parity<V_RING>(i), &sm.alone[0], nullptr, 0);
        for (int i = max(0, total - K_RING); i < total; ++i) mbar_wait_line(&sm.k_full[i % K_RING], (i / K_RING) & 1, &sm.alone[0], nullptr, 0);
        for (int i = max(0, n_items - 2); i < n_items; ++i) mbar_wait_line(&sm.q_full[slot<2>(i)], round_parity<2>(i), &sm.alone[0], nullptr, 0);
    }
    __syncwarp();
}

// P.V(g), into accumulator g & 1, as soon as P^(g) is delivered, V8(g) is there and the flush of tile g - 2 has read the
// accumulator.
__device__ __forceinline__ void pv_warp(AttSmem& sm, const AttArgs& a, int k_tiles, uint32_t tmem) {
    const uint64_t p_desc0 = smem_desc(smem_u32(sm.p[0]), QUERY_TILE * 16, 128), v_desc0 = smem_desc(smem_u32(sm.v[0]), HEAD_DIM * 16, 128);
    const int total = a.items.mine() * k_tiles;
#pragma unroll 1
    for (int g = 0; g < total; ++g) {
        mbar_wait_line(&sm.v_full[slot<V_RING>(g)], round_parity<V_RING>(g), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
        pv_sync(g);
        tc_fence_after();
        issue_pv(tmem + COL_ACC + slot<2>(g) * HEAD_DIM, desc_at(p_desc0, slot<P_RING>(g) * (P_BYTES / 16)), desc_at(v_desc0, slot<V_RING>(g) * (V_BYTES / 16)),
                 &sm.acc_full[slot<2>(g)]);
    }
    commit_elected(&sm.drain[1]);
    mbar_wait_line(&sm.drain[1], 0, &sm.alone[1], nullptr, 0);
    __syncwarp();
}

// ---------------------------------------------------------------------------------------------------------------------
// softmax: thread = query row; warpgroup `mine` takes the key tiles g = mine, mine + 2, ..

__device__ __forceinline__ float load_scale(const float* p) {  // volatile: the compiler would otherwise sink the load to its use, a tile later
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
// One key tile: scores -> P^ bytes in shared memory, (tile maximum, row sum) -> the flush threads.
// Returns whether the scores of this warpgroup's next tile were complete when the exponentials began.
// c: scores to the log2 domain; valid: keys of the tile that exist (MASKED).
template <bool V_TOKEN, bool MASKED>
__device__ __forceinline__ bool softmax_tile(AttSmem& sm, uint32_t ts, int g, int row, float c, int valid,
                                             const uint32_t (&magic)[FILL_BLOCK]) {
    const float2 c2 = make_float2(c, c), minus_magic = make_float2(-MAGIC, -MAGIC), plus_magic = make_float2(MAGIC, MAGIC), p_unit = make_float2(P_UNIT, P_UNIT);
    const float4* log_s4 = reinterpret_cast<const float4*>(sm.tok[slot<V_RING>(g)]);
    const float4* inv_s4 = reinterpret_cast<const float4*>(sm.tok[slot<V_RING>(g)] + KEY_TILE);
    uint8_t* p_row = sm.p[slot<P_RING>(g)] + row * 16;
    // The row's 64 scores, read once and kept in registers; the buffer goes back to its start value for S(g + S_RING) at once.
    float2 x[KEY_TILE / 16][8];
    tmem_ld64_sync(ts, reinterpret_cast<float2(&)[KEY_TILE / 2]>(x));
    tmem_fill<KEY_TILE>(ts, magic);
    float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int step = 0; step < KEY_TILE / 16; ++step) {
        float2(&y)[8] = x[step];
        if (V_TOKEN) {  // log2 s_j joins the scores before the maximum
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float4 l = log_s4[step * 4 + j / 2];
                y[j] = fma2(add2(y[j], minus_magic), c2, make_float2(l.x, l.y));
                y[j + 1] = fma2(add2(y[j + 1], minus_magic), c2, make_float2(l.z, l.w));
            }
        }
        if (MASKED) {  // keys past the end: below every real score (|score| < 2^21)
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (step * 16 + j >= valid) (j % 2 ? y[j / 2].y : y[j / 2].x) = V_TOKEN ? -INFINITY : MAGIC - 4194303.0f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) top[j % 4] = max3(top[j % 4], y[j].x, y[j].y);
    }
    tmem_wait_st();
    tc_fence_before();
    s_free_arrive(g);
    float tile_max = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
    if (!V_TOKEN) tile_max = (tile_max - MAGIC) * c;
    // P^ = rint(255 * 2^(score * c - tile max)).  Per channel the float read back is MAGIC + score, so the exponent is
    // x * c + (offset - MAGIC * c) in ONE fused multiply-add; what the rounding of that constant loses (it is about
    // 2^11 in size) is put back exactly: `low` is the lost part, and the product p * 2^low happens inside the
    // multiply-add that rounds p to a byte.  Per token nothing is to be put back, and p times 2^-149 rounds it as well: the bits of
    // that denormal float are the integer, and two of them are packed into 16 bits by an exact multiply-add, which saves an
    // instruction per four bytes (22.87 -> 22.66 ms at 40 heads x 32760 tokens).  The exponent's argument itself ends below 8, where a float's step is 2^-21 (four
    // times that with a factor of 2^-23 taken into it to scale P^ on its way: 1.3e-5 of the bytes 1 .. 64 then missed their
    // exact rounding, 2.7e-6 so).
    const float offset = LOG2_255 - tile_max;
    float2 base2 = make_float2(offset, offset), k2 = make_float2(1.0f, 1.0f);
    if (!V_TOKEN) {
        const float a_hi = __fmul_rn(-MAGIC, c), a_lo = __fmaf_rn(-MAGIC, c, -a_hi);  // -MAGIC * c = a_hi + a_lo exactly
        const float sum = __fadd_rn(a_hi, offset), bb = __fsub_rn(sum, a_hi);
        const float low = __fadd_rn(__fadd_rn(__fsub_rn(a_hi, __fsub_rn(sum, bb)), __fsub_rn(offset, bb)), a_lo);  // a_hi + offset = sum + ..
        const float k = __fmaf_rn(low, 0.693147181f, 1.0f);  // 2^low, |low| < 2^-12
        base2 = make_float2(sum, sum), k2 = make_float2(k, k);
    }
    // (mbarrier.try_wait may hold the warp for microseconds when the phase is not complete, and after an item's last tiles
    // nothing comes: 4 heads x 1024 tokens took 22.3 us with it here and below, 14.4 without.)
    const bool asked = mbar_test(&sm.s_full[slot<S_RING>(g + 2)], round_parity<S_RING>(g + 2));
    unsigned isum[2] = {0, 0};
    float2 fsum = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int step = 0; step < KEY_TILE / 16; ++step) {
        float2(&y)[8] = x[step];
        float2 e[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = V_TOKEN ? add2(y[j], base2) : fma2(y[j], c2, base2);
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = make_float2(ex2(e[j].x), ex2(e[j].y));
        if (V_TOKEN) {  // the denominator sums p / s_j before rounding
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float4 r = inv_s4[step * 4 + j / 2];
                fsum = fma2(e[j], make_float2(r.x, r.y), fsum);
                fsum = fma2(e[j + 1], make_float2(r.z, r.w), fsum);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = V_TOKEN ? mul2(e[j], p_unit) : fma2(e[j], k2, plus_magic);  // the low byte of each is rint(p)
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (V_TOKEN) {
                const float2 two = fma2(e[2 * i + 1], make_float2(256.0f, 256.0f), e[2 * i]);  // exact: keys 0 and 2 | keys 1 and 3
                w[i] = __byte_perm(__float_as_uint(two.x), __float_as_uint(two.y), 0x5140);
            } else {
                const uint32_t lo = __byte_perm(__float_as_uint(e[2 * i].x), __float_as_uint(e[2 * i].y), 0x0040);
                const uint32_t hi = __byte_perm(__float_as_uint(e[2 * i + 1].x), __float_as_uint(e[2 * i + 1].y), 0x0040);
                w[i] = __byte_perm(lo, hi, 0x5410);
            }
            if (!V_TOKEN && MASKED) {  // keys past the end weigh nothing
                const int left = valid - (step * 16 + i * 4);
                w[i] = left >= 4 ? w[i] : left <= 0 ? 0u : (w[i] & ((1u << (8 * left)) - 1u));
            }
            isum[i % 2] = __dp4a(w[i], 0x01010101u, isum[i % 2]);
        }
        *reinterpret_cast<uint4*>(p_row + step * (QUERY_TILE * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (V_TOKEN) sm.p_sum[slot<ST_RING>(g)][row] = uint16_t(isum[0] + isum[1]);
    sm.st[slot<ST_RING>(g)][row] = make_float2(tile_max, V_TOKEN ? fsum.x + fsum.y : __uint2float_rn(isum[0] + isum[1]));
    fence_proxy_async();
    __syncwarp();
    pv_arrive(g);  // P^(g) and its record delivered
    return asked;
}

template <bool V_TOKEN>
__device__ __forceinline__ void softmax_warps(AttSmem& sm, const AttArgs& a, int k_tiles, uint32_t tmem, int warp, int row) {
    const int mine = warp / 4, in_group = warp % 4;
    const bool ragged = a.n_keys % KEY_TILE != 0;  // the last key tile of a head needs masking
    // The score buffers start at MAGIC_BITS, so what comes back from tensor memory is already a float (common.cuh).
    uint32_t magic[FILL_BLOCK];
    fill_block_init(magic, MAGIC_BITS);
    const uint32_t t_s = tmem + (uint32_t(in_group * 32) << 16) + COL_S;
#pragma unroll
    for (int b = 0; b < S_RING; b += 2) tmem_fill<KEY_TILE>(t_s + (mine + b) * KEY_TILE, magic);
    tmem_wait_st();
    tc_fence_before();
#pragma unroll
    for (int b = 0; b < S_RING; b += 2) s_free_arrive(mine + b);

    // The scale of this warpgroup's next key tile is loaded a whole tile ahead of its use.
    auto scale_at = [&](int item, int t) { return a.k_scale + size_t(a.items.head(item)) * k_tiles + t; };
    int g = mine, first = mine;  // key tile of the block; the item's first key tile of this warpgroup
    int item = blockIdx.x;
    bool asked = false;  // this warpgroup's next scores have been seen complete: asked while the tile before is under way
    float sk = first < k_tiles ? load_scale(scale_at(item, first)) : 0.0f;
    for (; item < a.items.count; item += gridDim.x) {
        const float* sk_head = scale_at(item, 0);
        const float sq = a.q_scale[size_t(a.items.head(item)) * a.items.allocated + a.items.tile(item)];
        const int next_first = (first + k_tiles) & 1;  // in the block's next item
        const bool more = item + int(gridDim.x) < a.items.count;
        if (first >= k_tiles && more) sk = load_scale(scale_at(item + gridDim.x, next_first));  // (one key tile per head: the other warpgroup has this item)
#pragma unroll 1
        for (int t = first; t < k_tiles; t += 2, g += 2) {
            const float c = (sq * sk) * a.scale_log2;
            if (t + 2 < k_tiles)
                sk = load_scale(sk_head + t + 2);
            else if (more && next_first < k_tiles)
                sk = load_scale(scale_at(item + gridDim.x, next_first));
            // the scores are there, and P.V(g - P_RING) has read the P^ image this tile's goes into
            if (g >= P_RING) p_free_sync(g);
            const bool there = asked || mbar_wait_line(&sm.s_full[slot<S_RING>(g)], round_parity<S_RING>(g), &sm.abort_flag, a.status, STATUS_WAIT_SCORES);
            // Per token: the keys' scales came with the V tile, usually long ago
            if (V_TOKEN && there) mbar_wait_line(&sm.v_full[slot<V_RING>(g)], round_parity<V_RING>(g), &sm.abort_flag, a.status, STATUS_WAIT_TILE);
            __syncwarp();
            tc_fence_after();
            const uint32_t ts = t_s + slot<S_RING>(g) * KEY_TILE;
            if (ragged && t + 1 == k_tiles)
                asked = softmax_tile<V_TOKEN, true>(sm, ts, g, row, c, a.n_keys - t * KEY_TILE, magic);
            else
                asked = softmax_tile<V_TOKEN, false>(sm, ts, g, row, c, KEY_TILE, magic);
        }
        first = next_first;
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// flush: thread = query row, the row's 128 sums in registers

// The outlier keys were zeros in V8: their exact share p * v / v_scale, with p = 255 * 2^(score - final max), from this
// row's Q^ (still in shared memory) and the key's K^ row and scale (csrc/flash.cu:748-790).  The keys' K^ rows and V rows
// are the same for all 128 rows: the flush warps bring them into the staging rows, sixteen outliers at a time, and meet at
// a barrier of their own.
__device__ __forceinline__ void add_outliers(AttSmem& sm, const AttArgs& a, int k_tiles, int head, int q_tile, int q_slot, int row, float m,
                                             float2 (&o)[HEAD_DIM / 2]) {
    static_assert(OUTLIER_BATCH * (HEAD_DIM * 4 + HEAD_DIM + 4) <= int(sizeof(sm.staged)), "the staging rows hold a batch of outlier rows");
    uint8_t* batch = reinterpret_cast<uint8_t*>(sm.staged);
    float* rows_s = reinterpret_cast<float*>(batch);                                    // [OUTLIER_BATCH][128]
    uint4* k_rows_s = reinterpret_cast<uint4*>(batch + OUTLIER_BATCH * HEAD_DIM * 4);  // [OUTLIER_BATCH][8]: the key's 128 codes
    int* keys_s = reinterpret_cast<int*>(batch + OUTLIER_BATCH * HEAD_DIM * 5);        // [OUTLIER_BATCH], -1: no such key
    const float sq = a.q_scale[size_t(head) * a.items.allocated + q_tile];
    const float* sk = a.k_scale + size_t(head) * k_tiles;
    const uint4* q_row8 = reinterpret_cast<const uint4*>(sm.q[q_slot] + row * 16);  // chunk c: QUERY_TILE uint4 further
    for (int i0 = 0; i0 < a.n_outliers; i0 += OUTLIER_BATCH) {
        const int n = min(OUTLIER_BATCH, a.n_outliers - i0);
        asm volatile("bar.sync %0, 128;" ::"n"(BAR_FLUSH) : "memory");  // the batch before has been used, the item before has left the staging rows
        for (int piece = row; piece < n * (HEAD_DIM / 4); piece += 128)
            reinterpret_cast<float4*>(rows_s)[piece] = reinterpret_cast<const float4*>(a.outlier_rows + (size_t(head) * a.n_outliers + i0) * HEAD_DIM)[piece];
        for (int piece = row; piece < n * (HEAD_DIM / 16); piece += 128) {
            const int i = piece / (HEAD_DIM / 16), c = piece % (HEAD_DIM / 16);
            const int key = a.outlier_keys[size_t(head) * a.n_outliers + i0 + i];
            const bool there = key >= 0 && key < a.n_keys;
            k_rows_s[piece] = there ? reinterpret_cast<const uint4*>(a.k8 + (size_t(head) * k_tiles + key / KEY_TILE) * K_BYTES + (key % KEY_TILE) * 16)[c * KEY_TILE]
                                    : make_uint4(0, 0, 0, 0);
            if (c == 0) keys_s[i] = there ? key : -1;
        }
        asm volatile("bar.sync %0, 128;" ::"n"(BAR_FLUSH) : "memory");
        for (int i = 0; i < n; ++i) {
            const int key = keys_s[i];
            if (key < 0) continue;
            int dot = 0;
#pragma unroll
            for (int c = 0; c < HEAD_DIM / 16; ++c) {
                const uint4 qv = q_row8[c * QUERY_TILE], kv = k_rows_s[i * (HEAD_DIM / 16) + c];
                dot = __dp4a(int(qv.x), int(kv.x), dot);
                dot = __dp4a(int(qv.y), int(kv.y), dot);
                dot = __dp4a(int(qv.z), int(kv.z), dot);
                dot = __dp4a(int(qv.w), int(kv.w), dot);
            }
            const float p = ex2(__int2float_rn(dot) * ((sq * sk[key / KEY_TILE]) * a.scale_log2) - m) * (255.0f * SUM_UNIT);
            const float2 p2 = make_float2(p, p);
            const float2* v_row = reinterpret_cast<const float2*>(rows_s + i * HEAD_DIM);
#pragma unroll
            for (int j = 0; j < HEAD_DIM / 2; ++j) o[j] = fma2(p2, v_row[j], o[j]);
        }
    }
    asm volatile("bar.sync %0, 128;" ::"n"(BAR_FLUSH) : "memory");  // the last batch has been used: the staging rows may take output
}

template <bool V_TOKEN, bool OUTLIERS>
__device__ __forceinline__ void flush_warps(AttSmem& sm, const AttArgs& a, int k_tiles, uint32_t tmem, int warp, int row) {
    const int lane = row % 32;
    const uint32_t t_acc = tmem + (uint32_t(warp * 32) << 16) + COL_ACC;
    uint8_t* staged = sm.staged[warp];
    const int total = a.items.mine() * k_tiles;
    for (int b = 0; b < min(2, total); ++b) pv_arrive(b);  // the accumulators are free to begin with
    int g = 0, i = 0;
    float2 o[HEAD_DIM / 2], y[2][16];
    // The tiles' accumulators come in four pieces of 32 channels through two sets of registers: while one piece is added up
    // the next is on its way, also from one tile to the next if its P.V is complete by then.
    // P.V(g) was issued after the softmax of tile g had delivered its record, so where the accumulator is, the record is too.
    auto load = [&](int tile, int piece, float2(&into)[16]) { tmem_ld32_async(t_acc + slot<2>(tile) * HEAD_DIM + piece * 32, into); };
    auto wait_for = [&](int tile) {
        const bool there = mbar_wait_line(&sm.acc_full[slot<2>(tile)], round_parity<2>(tile), &sm.abort_flag, a.status, STATUS_WAIT_PV);
        __syncwarp();
        tc_fence_after();
        return there;
    };
    bool ok = wait_for(0);
    load(0, 0, y[0]);
    float2 record = sm.st[0][row];  // tile maximum, row sum
    float p_sum = V_TOKEN ? float(sm.p_sum[0][row]) : 0.0f;
    auto next_record = [&](int tile) {
        record = sm.st[slot<ST_RING>(tile)][row];
        if (V_TOKEN) p_sum = float(sm.p_sum[slot<ST_RING>(tile)][row]);
    };

    for (int item = blockIdx.x; item < a.items.count; item += gridDim.x, ++i) {
        // `m` is the exponent the sums are kept at, not the running maximum: out = sum over tiles of 2^(tile max - m) *
        // acc, the same for the denominator, and the common factor cancels at the end.  The textbook form moves m to
        // every new maximum and multiplies out and den by 2^(m_old - m_new) each time; here m is the first tile's maximum and
        // moves only when a tile's is more than 2^REFERENCE_SLACK above it.
        float m = record.x, beta = 1.0f, den = 0.0f, bias = 0.0f;  // bias: what V8's bias has added to every sum since it was last taken out
#pragma unroll
        for (int j = 0; j < HEAD_DIM / 2; ++j) o[j] = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (int t = 0; t < k_tiles; ++t, ++g) {
            // Is the next tile's accumulator complete?  Asked now, looked at after the first piece: the answer takes some sixty
            // cycles.  (All lanes get the same one; the vote says so to the compiler.)  Its record is read then too, and its
            // factor is ready before this tile is done.  Here it pays to be held until the phase completes (1.060 ms per channel
            // for 37 heads x 8192 tokens, 1.324 per token; with a test 1.10 and 1.41): never for a tile that does not come.
            const bool more = g + 1 < total, asked = more && mbar_try(&sm.acc_full[slot<2>(g + 1)], round_parity<2>(g + 1));
            if (record.x > m + REFERENCE_SLACK) {
                const float alpha = ex2(m - record.x);
                m = record.x, beta = 1.0f;
                den *= alpha, bias *= alpha;
#pragma unroll
                for (int j = 0; j < HEAD_DIM / 2; ++j) o[j] = mul2(o[j], make_float2(alpha, alpha));
            }
            __syncwarp();
            // V8's sign; in the form that measured faster (40 heads x 32760 tokens: 17.82 ms against 18.09 per channel, 22.66
            // against 22.55 per token)
            const float signed_beta = V_TOKEN ? (t & 1 ? -beta : beta) : __uint_as_float(__float_as_uint(beta) ^ (uint32_t(t) << 31));
            const float2 beta2 = make_float2(signed_beta * BETA_UNIT, signed_beta * BETA_UNIT);
            bool next_there = false;
#pragma unroll
            for (int piece = 0; piece < 3; ++piece) {
                tmem_wait_ld();
                reg_fence16(y[piece % 2]);
                load(g, piece + 1, y[(piece + 1) % 2]);
                flush32(y[piece % 2], o + 16 * piece, beta2);
                reg_fence16(y[piece % 2]);
                if (piece == 0) {
                    den += record.y * beta;
                    bias += (V_TOKEN ? p_sum : record.y) * (signed_beta * (V8_BIAS * SUM_UNIT));
                    next_there = __all_sync(0xffffffffu, asked && more);
                    if (next_there) {
                        tc_fence_after();
                        next_record(g + 1);
                    }
                }
            }
            tmem_wait_ld();
            reg_fence16(y[1]);
            tc_fence_before();
            if (g + 2 < total) pv_arrive(g + 2);  // the accumulator has been read: P.V(g + 2) may overwrite it
            if (g + P_RING < total) p_free_arrive(g);
            if (next_there) load(g + 1, 0, y[0]);
            beta = ex2(record.x - m);
            flush32(y[1], o + 48, beta2);
            if (t % BIAS_TILES == BIAS_TILES - 1 || t + 1 == k_tiles) {
                const float2 bias2 = make_float2(-bias, -bias);
#pragma unroll
                for (int j = 0; j < HEAD_DIM / 2; ++j) o[j] = add2(o[j], bias2);
                bias = 0.0f;
            }
            if (more && !next_there) {
                ok &= wait_for(g + 1);
                load(g + 1, 0, y[0]);
                next_record(g + 1);
                beta = ex2(record.x - m);
            }
        }

        const int head = a.items.head(item), q_tile = a.items.tile(item);
        ok &= mbar_wait_line(&sm.q_full[slot<2>(i)], round_parity<2>(i), &sm.abort_flag, a.status, STATUS_WAIT_TILE);  // V's channel scales came with Q8
        ok = __all_sync(0xffffffffu, ok && !gave_up(sm.abort_flag));
        bulk_store_read_wait();  // the item before has left the staging rows
        if constexpr (OUTLIERS) {
            add_outliers(sm, a, k_tiles, head, q_tile, slot<2>(i), row, m, o);
        }
        // Out through shared memory: a thread writes its row there and one bulk copy takes the 256 bytes to the caller's tensor.
        const float inv = (1.0f / den) * (1.0f / SUM_UNIT);
        const float4* vs4 = reinterpret_cast<const float4*>(sm.v_scale[slot<2>(i)]);
        uint8_t* staged_row = staged + lane * STAGED_PITCH;
#pragma unroll
        for (int chunk = 0; chunk < HEAD_DIM / 8; ++chunk) {
            const float4 s0 = vs4[2 * chunk], s1 = vs4[2 * chunk + 1];
            const float2* v = o + chunk * 4;
            *reinterpret_cast<uint4*>(staged_row + chunk * 16) =
                make_uint4(output_pair(v[0].x * s0.x * inv, v[0].y * s0.y * inv, a.out_layout.half), output_pair(v[1].x * s0.z * inv, v[1].y * s0.w * inv, a.out_layout.half),
                           output_pair(v[2].x * s1.x * inv, v[2].y * s1.y * inv, a.out_layout.half), output_pair(v[3].x * s1.z * inv, v[3].y * s1.w * inv, a.out_layout.half));
        }
        send_staged_rows(staged, lane, q_tile * QUERY_TILE + warp * 32, a.n_queries, head, a.out, a.out_layout, a.peers, ok);
        if (lane == 0) mbar_arrive(&sm.q_free[slot<2>(i)]);  // Q8 and V's scales have been used
    }
    bulk_store_read_wait();
}

template <bool V_TOKEN, bool OUTLIERS>
__global__ void __launch_bounds__(ATT_THREADS, 1) attention_int8_kernel(const __grid_constant__ AttArgs a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    AttSmem& sm = *reinterpret_cast<AttSmem*>(smem_raw);
    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x / 32), 0), row = threadIdx.x % 128;  // (the shuffle tells the compiler that it is uniform)
    const int k_tiles = (a.n_keys + KEY_TILE - 1) / KEY_TILE;

    if (threadIdx.x == 0) {
        sm.abort_flag = 0;
        for (int& word : sm.alone) word = 0;
        for (int s = 0; s < 2; ++s) {
            mbar_init(&sm.q_full[s], 1), mbar_init(&sm.q_free[s], 5);  // the scores' instructions and the four flush warps
            mbar_init(&sm.acc_full[s], 1);
            mbar_init(&sm.drain[s], 1);
        }
        for (int s = 0; s < K_RING; ++s) mbar_init(&sm.k_full[s], 1);
        for (int s = 0; s < V_RING; ++s) mbar_init(&sm.v_full[s], 1);
        for (int s = 0; s < S_RING; ++s) mbar_init(&sm.s_full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == FLUSH_WARP) tmem_alloc(&sm.tmem_base, TMEM_COLUMNS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem_base, 0);
    wait_for_previous_kernel();

    if (warp >= FLUSH_WARP && warp < SOFTMAX_WARP) {
        set_registers<FLUSH_REGISTERS, LAUNCH_REGISTERS>();
        flush_warps<V_TOKEN, OUTLIERS>(own_view(sm), a, k_tiles, tmem, warp - FLUSH_WARP, row);
    } else if (warp >= SOFTMAX_WARP) {
        set_registers<SOFTMAX_REGISTERS, LAUNCH_REGISTERS>();
        softmax_warps<V_TOKEN>(own_view(sm), a, k_tiles, tmem, warp - SOFTMAX_WARP, row);
    } else {
        set_registers<SERVICE_REGISTERS, LAUNCH_REGISTERS>();
        if (warp == SCORES_WARP) {
            scores_warp<V_TOKEN>(own_view(sm), a, k_tiles, tmem);
        } else if (warp == PV_WARP) {
            pv_warp(own_view(sm), a, k_tiles, tmem);
        }
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x / 32 == FLUSH_WARP) {
        tc_fence_after();
        tmem_dealloc(sm.tmem_base, TMEM_COLUMNS);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Self-test: one tcgen05.mma chain on operand images given by the caller, accumulator copied out as it lies in tensor memory.

__global__ void __launch_bounds__(128) selftest_mma_i8_kernel(const uint8_t* __restrict__ a_image, const uint8_t* __restrict__ b_image,
                                                              int n, int k, int a_unsigned, int32_t* __restrict__ d, int* status) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t* a_s = smem_raw;             // [k / 16][128][16]
    uint8_t* b_s = smem_raw + 128 * k;   // [k / 16][n][16]
    __shared__ uint64_t done;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    for (int i = threadIdx.x; i < 128 * k / 16; i += 128) reinterpret_cast<uint4*>(a_s)[i] = reinterpret_cast<const uint4*>(a_image)[i];
    for (int i = threadIdx.x; i < n * k / 16; i += 128) reinterpret_cast<uint4*>(b_s)[i] = reinterpret_cast<const uint4*>(b_image)[i];
    if (threadIdx.x == 0) {
        abort_flag = 0;
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_proxy_async();
    if (threadIdx.x / 32 == 0) tmem_alloc(&tmem_base, 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (threadIdx.x == 0) {
        for (int ks = 0; ks < k / 32; ++ks) {
            const uint64_t a_desc = smem_desc(smem_u32(a_s) + ks * 2 * 128 * 16, 128 * 16, 128), b_desc = smem_desc(smem_u32(b_s) + ks * 2 * n * 16, n * 16, 128);
            if (a_unsigned == 2)  // kind::tf32: the images hold floats, k / 4 per row; an instruction takes 8 = 32 bytes of a row
                mma_tf32_ss(tmem, a_desc, b_desc, idesc_tf32(128, n), ks > 0);
            else
                mma_i8_ss(tmem, a_desc, b_desc, idesc_i8(!a_unsigned, 128, n), ks > 0);
        }
        mma_commit(&done);
    }
    const bool ok = mbar_wait(&done, 0, &abort_flag, status, STATUS_WAIT_SCORES);
    tc_fence_after();
    if (ok) {
        const uint32_t lane_base = uint32_t((threadIdx.x / 32) * 32) << 16;
        for (int c0 = 0; c0 < n; c0 += 32) {
            uint32_t r[32];
            tmem_ld32(tmem + lane_base + c0, r);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) d[threadIdx.x * n + c0 + i] = int32_t(r[i]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x / 32 == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

}  // namespace unica

using namespace unica;

int unica_attention_int8(const int8_t* q8, const float* q_scale, const int8_t* k8, const float* k_scale, const int8_t* v8,
                          const float* v_scale, const float* v_token, int v_mode, const int* outlier_keys, const float* outlier_rows,
                          int n_outliers, void* out, void* const* peer_out, int n_peers, unica_token_layout out_layout, int heads,
                          int n_queries, int n_keys, float scale_log2, int* status, void* stream, bool overlapped) {
    if (!q8 || !q_scale || !k8 || !k_scale || !v8 || !v_scale || !out) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_int8: null pointer");
    if (heads <= 0 || heads > 65535 || n_queries <= 0 || n_keys <= 0)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_int8: heads must be in 1..65535, n_queries and n_keys positive");
    if (v_mode != UNICA_B200_V_CHANNEL && v_mode != UNICA_B200_V_TOKEN && v_mode != UNICA_B200_V_OUTLIERS)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_int8: unknown v_mode");
    if (v_mode == UNICA_B200_V_OUTLIERS && (!outlier_keys || !outlier_rows || n_outliers < 1 || n_outliers > 8))
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_int8: the outliers mode needs outlier_keys, outlier_rows and 1..8 outliers");
    if (v_mode == UNICA_B200_V_TOKEN && !v_token) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_int8: per-token mode needs v_token");
    PeerOutputs peers = {};
    if (int e = unica_peer_outputs(out, peer_out, n_peers, &peers)) return e;
    if (int e = unica_check_device()) return e;
    AttArgs args = {};
    args.q8 = q8, args.k8 = k8, args.v8 = v8, args.q_scale = q_scale, args.k_scale = k_scale, args.v_scale = v_scale, args.v_token = v_token;
    args.outlier_keys = outlier_keys, args.outlier_rows = outlier_rows, args.n_outliers = n_outliers;
    args.out = static_cast<__nv_bfloat16*>(out), args.out_layout = to_layout(out_layout), args.peers = peers;
    args.n_queries = n_queries, args.n_keys = n_keys, args.scale_log2 = scale_log2, args.status = status;
    const long long tiles = (n_queries + QUERY_TILE - 1) / QUERY_TILE, count = tiles * heads;
    if (count > INT_MAX / 2) return unica_fail(UNICA_B200_ERR_ARGUMENT, "attention_int8: more than 2^30 tiles of 128 queries");
    args.items.tiles = int(tiles), args.items.allocated = int(tiles + 1) / 2 * 2, args.items.count = int(count);  // Q8 holds an even number of tiles
    const size_t smem = sizeof(AttSmem) + 128;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto launch = [&](auto kernel, int instance) -> int {
        // Set up once per kernel instance and device: the shared-memory size, and a check that the build holds the
        // registers its setmaxnreg split needs (setmaxnreg only moves registers the block already has: asking for more
        // than the launch gives would make the flush warps wait for ever).
        constexpr int MAX_DEVICES = 64;
        static std::atomic<int> blocks_of[3][MAX_DEVICES];  // persistent blocks (one per SM), 0: not set up; the three instances share this lambda's one instantiation
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess) return unica_check_launch("attention_int8 (device)");
        int blocks = device < MAX_DEVICES ? blocks_of[instance][device].load(std::memory_order_acquire) : 0;
        if (blocks == 0) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess ||
                cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess)
                return unica_check_launch("attention_int8 (shared memory size)");
            cudaFuncAttributes attributes;
            if (cudaFuncGetAttributes(&attributes, kernel) != cudaSuccess) return unica_check_launch("attention_int8 (attributes)");
            if (attributes.numRegs * ATT_THREADS < 128 * (2 * SOFTMAX_REGISTERS + FLUSH_REGISTERS + SERVICE_REGISTERS))
                return unica_fail(UNICA_B200_ERR_KERNEL, "attention_int8: this build holds fewer registers per block than its setmaxnreg split needs");
            if (cudaDeviceGetAttribute(&blocks, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return unica_check_launch("attention_int8 (device)");
            if (device < MAX_DEVICES) blocks_of[instance][device].store(blocks, std::memory_order_release);
        }
        launch_after(kernel, dim3(args.items.count < blocks ? args.items.count : blocks), ATT_THREADS, smem, s, overlapped, args);
        return unica_check_launch("attention_int8");
    };
    return v_mode == UNICA_B200_V_TOKEN      ? launch(attention_int8_kernel<true, false>, 1)
           : v_mode == UNICA_B200_V_OUTLIERS ? launch(attention_int8_kernel<false, true>, 2)
                                             : launch(attention_int8_kernel<false, false>, 0);
}

extern "C" int unica_b200_attention_int8(const int8_t* q8, const float* q_scale, const int8_t* k8, const float* k_scale,
                                         const int8_t* v8, const float* v_scale, const float* v_token, int v_mode,
                                         const int* outlier_keys, const float* outlier_rows, int n_outliers, void* out,
                                         unica_token_layout out_layout, int heads, int n_queries, int n_keys, float scale_log2,
                                         int* status, void* stream) {
    return unica_attention_int8(q8, q_scale, k8, k_scale, v8, v_scale, v_token, v_mode, outlier_keys, outlier_rows, n_outliers, out, nullptr, 0,
                          out_layout, heads, n_queries, n_keys, scale_log2, status, stream);
}

extern "C" int unica_b200_attention_int8_peers(const int8_t* q8, const float* q_scale, const int8_t* k8, const float* k_scale,
                                               const int8_t* v8, const float* v_scale, const float* v_token, int v_mode,
                                               const int* outlier_keys, const float* outlier_rows, int n_outliers, void* out,
                                               void* const* peer_out, int n_peers, unica_token_layout out_layout, int heads,
                                               int n_queries, int n_keys, float scale_log2, int* status, void* stream) {
    return unica_attention_int8(q8, q_scale, k8, k_scale, v8, v_scale, v_token, v_mode, outlier_keys, outlier_rows, n_outliers, out, peer_out,
                          n_peers, out_layout, heads, n_queries, n_keys, scale_log2, status, stream);
}

extern "C" int unica_b200_selftest_mma_i8(const void* a_image, const void* b_image, int n, int k, int a_unsigned, int variant,
                                          int32_t* d, void* stream) {
    if (!a_image || !b_image || !d) return unica_fail(UNICA_B200_ERR_ARGUMENT, "selftest_mma_i8: null pointer");
    if (n < 32 || n > 128 || n % 32 || k < 32 || k > 128 || k % 32)
        return unica_fail(UNICA_B200_ERR_ARGUMENT, "selftest_mma_i8: n and k must be multiples of 32 in 32..128");
    if (variant != 0) return unica_fail(UNICA_B200_ERR_ARGUMENT, "selftest_mma_i8: variant must be 0");
    if (int e = unica_check_device()) return e;
    const size_t smem = size_t(128 + n) * k + 128;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int* status = nullptr;
    if (cudaMalloc(&status, sizeof(int)) != cudaSuccess || cudaMemsetAsync(status, 0, sizeof(int), s) != cudaSuccess) {
        const int e = unica_check_launch("selftest_mma_i8 (status word)");
        cudaFree(status);  // a no-op when the allocation itself failed
        return e;
    }
    selftest_mma_i8_kernel<<<1, 128, smem, s>>>(static_cast<const uint8_t*>(a_image), static_cast<const uint8_t*>(b_image), n, k,
                                                a_unsigned, d, status);
    int host_status = 0;
    cudaError_t e = cudaMemcpyAsync(&host_status, status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(status);
    if (e != cudaSuccess) {
        unica_fail(UNICA_B200_ERR_CUDA, cudaGetErrorString(e));
        return UNICA_B200_ERR_CUDA;
    }
    if (host_status) return unica_fail(UNICA_B200_ERR_KERNEL, "selftest_mma_i8: the tensor-core instruction never completed");
    return UNICA_B200_OK;
}

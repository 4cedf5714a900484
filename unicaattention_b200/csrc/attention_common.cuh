// What the two attention kernels share: the register split between warpgroups, rings, the items of a persistent block, and the
// instructions that one elected lane of a warp issues.
#pragma once

#include "common.cuh"

namespace unica {

// REGISTERS per thread for this warpgroup, of the LAUNCH per thread that the block was launched with.
template <int REGISTERS, int LAUNCH>
__device__ __forceinline__ void set_registers() {  // every warp of a warpgroup executes it
    if constexpr (REGISTERS > LAUNCH)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGISTERS));
    else
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGISTERS));
}
// Tile g's slot in a ring of N, and the phase parity of the slot's barrier for it.
template <int N>
__device__ __forceinline__ int slot(int g) {
    static_assert((N & (N - 1)) == 0, "rings are powers of two: slots and parities are bits of the tile count");
    return g & (N - 1);
}
template <int N>
__device__ __forceinline__ int round_parity(int g) {
    return (g / N) & 1;
}
// What a block's items are: tiles of 128 query rows, head by head.
struct Items {
    int tiles, allocated, count;  // query tiles per head: with queries in them, and in Q8 (an even number); items of the call
    __device__ __forceinline__ int mine() const { return (count - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x); }  // of this block
    __device__ __forceinline__ int head(int item) const { return item / tiles; }
    __device__ __forceinline__ int tile(int item) const { return item % tiles; }
};

// The block's shared memory as one role sees it: an address the compiler cannot relate to the other roles' (it otherwise
// computes the addresses common to several roles before they part, and holds them in registers the computing loops need).
template <typename Smem>
__device__ __forceinline__ Smem& own_view(Smem& sm) {
    uint32_t base = smem_u32(&sm);
    asm volatile("" : "+r"(base));
    return *static_cast<Smem*>(__cvta_shared_to_generic(base));
}

// A descriptor `units` of 16 bytes further on in shared memory (its address is in the low word).
__device__ __forceinline__ uint64_t desc_at(uint64_t desc, uint32_t units) { return (desc & 0xffffffff00000000ull) | (uint32_t(desc) + units); }

__device__ __forceinline__ void commit_elected(uint64_t* bar) {
    asm volatile(
        "{\n\t"
        ".reg .pred e;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "}" ::"r"(smem_u32(bar))
        : "memory");
}

// A copy to shared memory whose arrival its barrier counts, issued by one elected lane of a converged warp.
__device__ __forceinline__ void copy_elected(void* dst, const void* src, int bytes, uint64_t* full) {
    asm volatile(
        "{\n\t"
        ".reg .pred e;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|e, 0xffffffff;\n\t"
        "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %2;\n\t"
        "@e cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t"
        "}" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(full))
        : "memory");
}

// Has a wait of any warp of the block given up?  Asked before an item's rows are stored: the warps that store them see their own waits
// only, and one that gave up goes on with whatever lies in its buffers.
__device__ __forceinline__ bool gave_up(const int& abort_flag) {
    int word;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(word) : "r"(smem_u32(&abort_flag)) : "memory");
    return word != 0;
}

// Output rows out through shared memory: each lane of a warp has written its row (256 bytes, STAGED_PITCH apart) and one bulk copy
// per row takes it to the caller's tensor.  bulk_store_read_wait() before the rows are written again.
constexpr int STAGED_PITCH = HEAD_DIM * 2 + 16;  // bytes from one staged output row to the next: rows of a quarter-warp on different banks
__device__ __forceinline__ void send_staged_rows(const uint8_t* staged, int lane, int first_row, int n_queries, int head, __nv_bfloat16* out,
                                                 const TokenLayout& layout, const PeerOutputs& peers, bool ok) {
    fence_proxy_async();
    if (ok && first_row + lane < n_queries) bulk_store(out + layout.offset(head, first_row + lane), staged + lane * STAGED_PITCH, HEAD_DIM * 2);
    bulk_store_commit();
    __syncwarp();
    if (peers.count > 0 && ok) {  // plain stores to other GPUs, two whole rows per instruction
        for (int pair = 0; pair < 16; ++pair) {
            const int r = 2 * pair + lane / 16;
            const uint4 value = *reinterpret_cast<const uint4*>(staged + r * STAGED_PITCH + (lane % 16) * 16);
            if (first_row + r < n_queries)
                for (int peer = 0; peer < peers.count; ++peer)
                    *reinterpret_cast<uint4*>(peers.out[peer] + layout.offset(head, first_row + r) + (lane % 16) * 8) = value;
        }
        __syncwarp();
    }
}

}  // namespace unica

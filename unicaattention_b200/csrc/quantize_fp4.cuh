// The NVFP4 quantizers' tile routines, shared by the one-tile-per-block kernels (quantize_fp4.cu) and the kernel that
// quantizes a whole short call in one launch (quantize_call.cu).
#pragma once

#include <cuda_fp8.h>

#include "quantize_int8.cuh"

namespace unica {

constexpr int FP4_THREADS = 256;
constexpr int V4_ROWS = 144;      // 128 channels + 16 rows of ones: their column of P.V is the running denominator
constexpr int V4_SF_WORDS = 256;  // scale words of a tile: two blocks of [32 lanes][4], the second for rows 128..143

__host__ __device__ __forceinline__ int slot_key(int k) { return 32 * (k / 32) + 8 * (k % 8 / 2) + 2 * (k % 32 / 8) + k % 2; }

__device__ __forceinline__ uint32_t to_e4m3(float x) { return __nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3); }
__device__ __forceinline__ float from_e4m3(uint32_t byte) {
    return __half2float(__half(__nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte), __NV_E4M3)));
}

// 8 floats -> 8 e2m1 codes, element i in nibble i.
__device__ __forceinline__ uint32_t pack_e2m1x8(const float* v) {
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
        : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
    return word;
}

// An outer scale and its reciprocal.  x / scale is taken without a division, by Markstein's correction step (see
// quotient_code2 in quantize_int8.cuh): bit for bit the IEEE quotient wherever it decides a code, given that the residual does
// not underflow (outer scales below 1e-27 take the division) and that the divisor's mantissa is not all ones.
struct Fp4Outer {
    float value, inverse;
    bool divide;
};
__device__ __forceinline__ Fp4Outer fp4_outer(float outer) { return Fp4Outer{outer, __frcp_rn(outer), outer < 1e-27f || needs_division(outer)}; }
__device__ __forceinline__ float2 quotient2(float2 x, float2 inv2, float2 minus_scale2) {
    const float2 q0 = mul2(x, inv2);
    return fma2(fma2(q0, minus_scale2, x), inv2, q0);
}

// One block of 16 values: scale byte and 16 codes (two words).
__device__ __forceinline__ void quantize_block16(float2 (&v)[8], const Fp4Outer& outer, uint32_t& byte, uint2& codes) {
    float amax = fmaxf(fabsf(v[0].x), fabsf(v[0].y));
#pragma unroll
    for (int i = 1; i < 8; ++i) amax = max3(amax, fabsf(v[i].x), fabsf(v[i].y));
    const float sixth = amax * (1.0f / 6.0f), q0 = sixth * outer.inverse;
    byte = to_e4m3(outer.divide ? __fdiv_rn(sixth, outer.value) : fmaf(fmaf(-q0, outer.value, sixth), outer.inverse, q0));
    const float scale = from_e4m3(byte) * outer.value;
    if (outer.divide || needs_division(scale)) {  // practically never
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = scale > 0.0f ? make_float2(__fdiv_rn(v[i].x, scale), __fdiv_rn(v[i].y, scale)) : make_float2(0.0f, 0.0f);
    } else {
        const float inv = scale > 0.0f ? __frcp_rn(scale) : 0.0f;  // a block whose scale is 0 holds zeros
        const float2 inv2 = make_float2(inv, inv), minus_scale2 = make_float2(-scale, -scale);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = quotient2(v[i], inv2, minus_scale2);
    }
    codes = make_uint2(pack_e2m1x8(&v[0].x), pack_e2m1x8(&v[4].x));
}

// Q or K minus its mean in NVFP4 along the channels: one tile of ROWS tokens (128: Q, 64: K) by a block of FP4_THREADS.
// SLOTS: row r of a tile holds token tile * 64 + slot_key(r) (K); else token tile * ROWS + r (Q).
// mean_of(token): the 128 means that go with the token, or null.
// codes: the tile's [4 chunks of 32 channels][ROWS][16] bytes; sf: Q [2 halves of 64 channels][32 lanes][4 words]
// [4] bytes, K [32 lanes][4 words][4] bytes (see the store below).
template <int ROWS, bool SLOTS, bool BY_ROW, typename MeanOf>
__device__ __forceinline__ void rows_fp4_tile(const __nv_bfloat16* __restrict__ x, const TokenLayout& in, MeanOf mean_of, const Fp4Outer& outer, int head,
                                              int tile, int n_tokens, uint8_t* __restrict__ tile_codes, uint8_t* __restrict__ tile_sf,
                                              const RopeTable& rope) {
    RowsRaw<ROWS, FP4_THREADS> raw;
    const __nv_bfloat16* first = x + in.offset(head, tile * ROWS);
#pragma unroll
    for (int it = 0; it < ROWS * 8 / FP4_THREADS; ++it) {
        const auto [row, block] = RowsItem<ROWS, FP4_THREADS, BY_ROW>(it);  // block of 16 channels
        const int at = SLOTS ? slot_key(row) : row;
        raw.piece[it][0] = raw.piece[it][1] = make_uint4(0, 0, 0, 0);
        if (tile * ROWS + at < n_tokens) {
            const __nv_bfloat16* src = first + at * in.token + block * 16;
            raw.piece[it][0] = load_bf16x8(src, in.half), raw.piece[it][1] = load_bf16x8(src + 8, in.half);
        }
    }
#pragma unroll
    for (int it = 0; it < ROWS * 8 / FP4_THREADS; ++it) {
        const auto [row, block] = RowsItem<ROWS, FP4_THREADS, BY_ROW>(it);
        const int token = SLOTS ? tile * ROWS + slot_key(row) : tile * ROWS + row;
        uint4 turns[2];  // the table's row, asked for under no condition: the compiler may then ask for several at once
        if (rope.table) {
            const uint4* f = reinterpret_cast<const uint4*>(rope.row(in, head, min(token, n_tokens - 1)) + block * 16);
            turns[0] = f[0], turns[1] = f[1];
        }
        float2 v[8];
        unpack8(raw.piece[it][0], reinterpret_cast<float2(&)[4]>(v[0]));
        unpack8(raw.piece[it][1], reinterpret_cast<float2(&)[4]>(v[4]));
        if (token < n_tokens) {
            if (rope.table) {  // rotate first: the mean is the rotated x's
                rope8(*reinterpret_cast<float(*)[8]>(v), turns[0]);
                rope8(*reinterpret_cast<float(*)[8]>(v + 4), turns[1]);
            }
            if (const float* mu = mean_of(token)) {
                const float4* m4 = reinterpret_cast<const float4*>(mu + block * 16);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 m = m4[i];
                    v[2 * i] = sub2(v[2 * i], make_float2(m.x, m.y)), v[2 * i + 1] = sub2(v[2 * i + 1], make_float2(m.z, m.w));
                }
            }
        }
        uint32_t byte;
        uint2 packed;
        quantize_block16(v, outer, byte, packed);
        *reinterpret_cast<uint2*>(tile_codes + ((block / 2) * ROWS + row) * 16 + (block % 2) * 8) = packed;
        // the word of (K step = block / 4, row): Q [2][32 lanes][4]: word row / 32 of lane row % 32; K [32 lanes][4]: word 2 step +
        // row / 32 of lane row % 32: the 16 bytes tcgen05.cp hands to one tensor-memory lane
        const int word = ROWS == 64 ? (row % 32) * 4 + 2 * (block / 4) + row / 32 : (block / 4) * ROWS + (row % 32) * 4 + row / 32;
        tile_sf[word * 4 + block % 4] = uint8_t(byte);
    }
}

// V in NVFP4 along the keys, per channel: one tile of 64 keys (slot order) by a block of FP4_THREADS.  low/high: the channel's
// min and max over the head ([128], this head's); v_outer [128] is written with tile 0.  tile: shared memory, free again after
// a __syncthreads().
// codes: the tile's [2 chunks of 32 slots][144 rows][16] bytes, rows 128..143 all ones (code 0x2);
// sf: [2 blocks][32 lanes][4 words] of 4 bytes: block 0 word c / 32 of lane c % 32 = channel c's four bytes, block 1 word 0 of
// lanes 0..15 = ones (0x38) for rows 128..143, zeros elsewhere.
using V4Tile = __nv_bfloat16[KEY_TILE][HEAD_DIM + 8];  // (rows 16-byte aligned)
__device__ __forceinline__ void v_fp4_load(VRaw& raw, const __nv_bfloat16* __restrict__ v, const TokenLayout& in, int head, int t, int n_tokens) {
    const int chunk = threadIdx.x % 16;
    const __nv_bfloat16* first = v + in.offset(head, t * KEY_TILE) + chunk * 8;
#pragma unroll
    for (int it = 0; it < KEY_TILE * 16 / FP4_THREADS; ++it) {
        const int key = slot_key(it * (FP4_THREADS / 16) + threadIdx.x / 16);
        raw.piece[it] = t * KEY_TILE + key < n_tokens ? load_bf16x8(first + key * in.token, in.half) : make_uint4(0, 0, 0, 0);
    }
}
__device__ __forceinline__ void v_fp4_finish(const VRaw& raw, const float* low, const float* high, int t, uint8_t* __restrict__ tile_codes,
                                             uint8_t* __restrict__ tile_sf, float* __restrict__ v_outer, V4Tile& tile) {  // by slot
#pragma unroll
    for (int it = 0; it < KEY_TILE * 16 / FP4_THREADS; ++it) {
        const int slot = it * (FP4_THREADS / 16) + threadIdx.x / 16, chunk = threadIdx.x % 16;
        *reinterpret_cast<uint4*>(&tile[slot][chunk * 8]) = raw.piece[it];
    }
    __syncthreads();
    for (int item = threadIdx.x; item < HEAD_DIM * 4; item += FP4_THREADS) {
        const int c = item % HEAD_DIM, block = item / HEAD_DIM;  // block of 16 slots
        const float outer = fmaxf(fmaxf(high[c], -low[c]) * (1.0f / 2688.0f), 1e-30f);
        if (t == 0 && block == 0) v_outer[c] = outer;
        float2 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = make_float2(__bfloat162float(tile[block * 16 + 2 * i][c]), __bfloat162float(tile[block * 16 + 2 * i + 1][c]));
        uint32_t byte;
        uint2 packed;
        quantize_block16(x, fp4_outer(outer), byte, packed);
        *reinterpret_cast<uint2*>(tile_codes + ((block / 2) * V4_ROWS + c) * 16 + (block % 2) * 8) = packed;
        tile_sf[((c % 32) * 4 + c / 32) * 4 + block] = uint8_t(byte);  // word c / 32 of lane c % 32
    }
    for (int item = threadIdx.x; item < 2 * 16 * 4; item += FP4_THREADS) {  // the rows of ones: 2 chunks x 16 rows x 4 words
        const int chunk = item / 64, row = 128 + item / 4 % 16, word = item % 4;
        reinterpret_cast<uint32_t*>(tile_codes + (chunk * V4_ROWS + row) * 16)[word] = 0x22222222u;
    }
    if (threadIdx.x < 128)  // second block: rows 128..143 (ones) are word 0 of lanes 0..15, the rest zeros
        reinterpret_cast<uint32_t*>(tile_sf)[128 + threadIdx.x] = threadIdx.x % 4 == 0 && threadIdx.x / 4 < 16 ? 0x38383838u : 0u;
}
__device__ __forceinline__ void v_fp4_tile(const __nv_bfloat16* __restrict__ v, const TokenLayout& in, const float* low, const float* high, int head, int t,
                                           int n_tokens, uint8_t* __restrict__ tile_codes, uint8_t* __restrict__ tile_sf, float* __restrict__ v_outer,
                                           V4Tile& tile) {
    VRaw raw;
    v_fp4_load(raw, v, in, head, t, n_tokens);
    v_fp4_finish(raw, low, high, t, tile_codes, tile_sf, v_outer, tile);
}

}  // namespace unica

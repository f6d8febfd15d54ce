// A 1 KB weight tile (16 rows x 256 inputs) times the int8 image of up to eight tokens on mma.m16n8k32: what the streaming
// product (gemv.cu) and the one-launch step of small TTT models (ttt_step.cu) share.
#pragma once

#include "bt_ptx.cuh"

namespace bt {

__device__ __forceinline__ void red_add_s32(int* p, int v) {
    asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(ptx::smem_u32(p)), "r"(v) : "memory");
}

__device__ __forceinline__ uint4 lds128(const void* p) { return *reinterpret_cast<const uint4*>(p); }

// One 1 KB tile: 2 A loads, 4 B loads, 32 ANDs, 8 MMAs.  The four field positions are four
// independent accumulator chains: their first MMAs are issued back to back, then the second.
// FIRST: the tile opens a row tile, its first MMAs start from the zero register (the
// accumulators need no clearing between row tiles).
template <bool FIRST>
__device__ __forceinline__ void tile_mma_r(int (&acc)[4][4], const uint4& w4, const uint4& v4, const uint4 (&b4)[4]) {
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const uint32_t mask = 0x03030303u << (2 * f);
        if (FIRST) ptx::mma_u8s8_zero(acc[f], w4.x & mask, v4.x & mask, w4.z & mask, v4.z & mask, b4[f].x, b4[f].z);
        else ptx::mma_u8s8(acc[f], w4.x & mask, v4.x & mask, w4.z & mask, v4.z & mask, b4[f].x, b4[f].z);
    }
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const uint32_t mask = 0x03030303u << (2 * f);
        ptx::mma_u8s8(acc[f], w4.y & mask, v4.y & mask, w4.w & mask, v4.w & mask, b4[f].y, b4[f].w);
    }
}

}  // namespace bt

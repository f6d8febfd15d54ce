// What the two prompt-attention kernels over a bf16 cache share (attn_dense.cu, attn_flash.cu).
#pragma once

#include "bt_dense.cuh"

namespace bt {

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// A raw score in units of ln 2, so that its exponential is one ex2: s * scale, or capped: cap * tanh(s * scale / cap) with
// tanh(u) = 1 - 2 / (e^2u + 1), whose absolute error is of the order of 1e-7 cap.
struct ScoreMap {
    float k, cap2;  // factor on the raw score; 2 cap / ln 2, 0: no cap
    __device__ __forceinline__ ScoreMap(float scale, float cap) {
        const float log2e = 1.4426950408889634f;
        k = cap > 0.0f ? scale / cap * (2.0f * log2e) : scale * log2e;
        cap2 = cap > 0.0f ? 2.0f * cap * log2e : 0.0f;
    }
    __device__ __forceinline__ float operator()(float s) const {
        const float u = s * k;
        return cap2 > 0.0f ? fmaf(-cap2, rcp(ex2(u) + 1.0f), 0.5f * cap2) : u;
    }
};
constexpr float kLn2 = 0.6931471805599453f;

// Latent attention: keys and values are bf16 rows expanded from the latents, the last key columns the rotated part all heads share.
struct LatentTile {
    const __nv_bfloat16* kv = nullptr;  // [sequence][kv_rows][heads k_main | heads v_stride]
    int64_t kv_ld = 0, kv_seq = 0;      // elements between positions and between sequences
    int k_main = 0;                     // columns of a head's own key part
    LatentView latent;
    int b0 = 0;
    const float* gate = nullptr;        // output gates of the rows
    int64_t gate_ld = 0;
};

// The tcgen05 form (attn_flash.cu); latent: lt describes keys and values, else the cache in a.kv does.
bool attn_flash_fits(const DenseAttn& a, bool latent);
cudaError_t launch_attn_flash(const DenseAttn& a, const LatentTile* lt, const ActOut& out, cudaStream_t s);

}  // namespace bt

// Small memory-bound kernels around the ternary products of one decode step:
// embedding gather, (RMSNorm | SwiGLU product | identity) + per-token int8 quantisation,
// dense bf16 lm_head, arg-max.  All f32 arithmetic; reference operation order is kept
// wherever a rounding could show (see each kernel).
#include "bt_common.cuh"
#include "bt_model.cuh"
#include "bt_ptx.cuh"

#include <type_traits>
namespace bt {

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_sum_i(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide reductions over blockDim.x threads (multiple of 32, <= 1024).
__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) red[w] = v;
    __syncthreads();
    float r = l < nw ? red[l] : 0.0f;
    r = warp_sum(r);
    __syncthreads();
    return r;
}
// REUSE = false: `red` is used by this one reduction only in the kernel, the closing barrier (which protects the
// array against the next use) is left out.
template <bool REUSE = true>
__device__ __forceinline__ float block_max(float v, float* red) {
    v = warp_max(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) red[w] = v;
    __syncthreads();
    float r = l < nw ? red[l] : 0.0f;
    r = warp_max(r);
    if (REUSE) __syncthreads();
    return r;
}
template <bool REUSE = true>
__device__ __forceinline__ double block_sum_d(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) red[w] = v;
    __syncthreads();
    double r = l < nw ? red[l] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (REUSE) __syncthreads();
    return r;
}
__device__ __forceinline__ int block_sum_i(int v, int* red) {
    v = warp_sum_i(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) red[w] = v;
    __syncthreads();
    int r = l < nw ? red[l] : 0;
    r = warp_sum_i(r);
    __syncthreads();
    return r;
}

// Two packed 16-bit weights -> f32: bf16 by shifting into the high half, IEEE half by conversion.
template <bool F16>
__device__ __forceinline__ void unpack16(uint32_t u, float& lo, float& hi) {
    if (F16) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
        lo = f.x; hi = f.y;
    } else {
        lo = __uint_as_float(u << 16);
        hi = __uint_as_float(u & 0xffff0000u);
    }
}

// ---------------------------------------------------------------------------------------
// embedding gather: h[b, :] = table[token[b], :]   (Embedding::forward, model/llama.rs:208)
// ---------------------------------------------------------------------------------------
__global__ void embed_kernel(const int32_t* __restrict__ tokens, const __nv_bfloat16* __restrict__ table,
                             int hidden, int vocab, float* __restrict__ h, unsigned int* __restrict__ clear,
                             int n_clear, bool f16) {
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const int b = blockIdx.x;
    if (b == 0)
        for (int i = threadIdx.x; i < n_clear; i += blockDim.x) clear[i] = 0u;
    int tok = tokens[b];
    tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
    const __nv_bfloat16* row = table + (int64_t)tok * hidden;
    float* out = h + (int64_t)b * hidden;
    // Eight values a thread and load.  A value at a time (hidden / 256 loads in turn, each a trip to device memory) a token of
    // 4096 values took 8.9 us, the first of a step's serial latencies (eight steps of decode, 8B shape, batch 1: 2 038 -> 2 015 us with this).
    if (((reinterpret_cast<uintptr_t>(row) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 && hidden % 8 == 0) {
#pragma unroll 2
        for (int c = 8 * threadIdx.x; c < hidden; c += 8 * blockDim.x) {
            const uint4 pk = __ldg(reinterpret_cast<const uint4*>(row + c));
            const uint32_t u[4] = {pk.x, pk.y, pk.z, pk.w};
            float f[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (f16) unpack16<true>(u[j], f[2 * j], f[2 * j + 1]);
                else unpack16<false>(u[j], f[2 * j], f[2 * j + 1]);
            }
            *reinterpret_cast<float4*>(out + c) = make_float4(f[0], f[1], f[2], f[3]);
            *reinterpret_cast<float4*>(out + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
        }
        return;
    }
    if (f16) {  // the table holds IEEE half values (a converted checkpoint's dtype)
        const __half* hrow = reinterpret_cast<const __half*>(row);
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) out[c] = __half2float(hrow[c]);
    } else {
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) out[c] = __bfloat162float(row[c]);
    }
}

// ---------------------------------------------------------------------------------------
// row transform + absmax int8 quantisation, one CTA per token, the row held in shared
// memory so that global memory is read once.
//   PRE_NONE   : v = x
//   PRE_RMSNORM: v = (x / sqrt(mean(x^2) + eps)) * w        (layers/rms_norm.rs:40-55)
//   PRE_SWIGLU : v = silu(gate) * up, x = gate and up interleaved in groups of 8 (the row order of the fused
//                gate|up projection: x[16 j + r] = gate[8 j + r], x[16 j + 8 + r] = up[8 j + r])  (layers/swiglu.rs:31-33)
// then s = max|v|/127, q = clamp(round(v * (127/max|v|))), sum_k q.  `v_out` (optional) receives v.
// ---------------------------------------------------------------------------------------
// Four consecutive floats; `vec` = the address is 16-byte aligned (uniform over the block).
__device__ __forceinline__ float4 load4(const float* p, bool vec) {
    if (vec) return *reinterpret_cast<const float4*>(p);
    return make_float4(p[0], p[1], p[2], p[3]);
}
// The same from bf16 values (`vec` = 16-byte aligned row start; a group of four is then 8-byte aligned).
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p, bool vec) {
    if (vec) {
        const uint2 u = *reinterpret_cast<const uint2*>(p);
        return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                           __uint_as_float(u.y & 0xffff0000u));
    }
    return make_float4(__bfloat162float(p[0]), __bfloat162float(p[1]), __bfloat162float(p[2]), __bfloat162float(p[3]));
}

// k must be a multiple of 4 (the packed weight layouts require it anyway).  A thread works on groups of four
// consecutive values; in the tensor-core layout these are the four residues of one k' (see gemm_tc_act_offset),
// which are first laid out in shared memory in the order of that layout's 16-byte pieces and then copied out a
// piece per thread.
template <int PRE, typename T = float>
__global__ void __launch_bounds__(1024) row_quant_kernel(const T* __restrict__ x, int64_t x_stride,
                                                         const float* __restrict__ w, float eps, int k,
                                                         int8_t* __restrict__ q, int64_t q_stride,
                                                         float* __restrict__ s_out,
                                                         int32_t* __restrict__ qsum_out,
                                                         float* __restrict__ v_out, int8_t* __restrict__ qtc,
                                                         int tc_nt, int k_tiles,
                                                         const unsigned int* __restrict__ amax_in,
                                                         unsigned int* __restrict__ amax_out) {
    // amax_in : [rows] bit patterns of max|v| to quantise with (a maximum agreed over several GPUs) instead of
    //           this row's own.  amax_out: values-only mode, the row's v goes to v_out and its max|v| (bits) to
    //           amax_out[row]; nothing is quantised.
    extern __shared__ __align__(16) float row[];  // k floats, then k_tiles * 256 staged bytes (tensor-core layout only)
    __shared__ float red_f[32];
    __shared__ double red_d[32];
    __shared__ int red_i[32];
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();  // a product launched behind this kernel may fetch its weights meanwhile
    const int b = blockIdx.x;
    const T* xr = x + (int64_t)b * x_stride;
    const bool xvec = ((reinterpret_cast<uintptr_t>(xr) & 15) == 0);
    const bool wvec = PRE == PRE_RMSNORM && ((reinterpret_cast<uintptr_t>(w) & 15) == 0);
    const int groups = k >> 2;
    float amax = 0.0f;
    if (PRE == PRE_RMSNORM) {
        // sum of squares in f64, rounded once: reproducible against the CPU restatement
        double ss = 0.0;
        for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
            const float4 v = load4(xr + 4 * gi, xvec);
            *reinterpret_cast<float4*>(row + 4 * gi) = v;
            ss = fma((double)v.x, (double)v.x, ss);
            ss = fma((double)v.y, (double)v.y, ss);
            ss = fma((double)v.z, (double)v.z, ss);
            ss = fma((double)v.w, (double)v.w, ss);
        }
        ss = block_sum_d<false>(ss, red_d);
        const float denom = sqrtf(__fadd_rn((float)(ss / (double)k), eps));
        for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
            float4 v = *reinterpret_cast<const float4*>(row + 4 * gi);  // written by this same thread
            const float4 ww = load4(w + 4 * gi, wvec);
            v.x = __fmul_rn(__fdiv_rn(v.x, denom), ww.x);
            v.y = __fmul_rn(__fdiv_rn(v.y, denom), ww.y);
            v.z = __fmul_rn(__fdiv_rn(v.z, denom), ww.z);
            v.w = __fmul_rn(__fdiv_rn(v.w, denom), ww.w);
            *reinterpret_cast<float4*>(row + 4 * gi) = v;
            amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
    } else if (PRE == PRE_SWIGLU) {
        for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
            const int c = 4 * gi;  // outputs c .. c + 3: gate at x[16 (c / 8) + c % 8 ..], up 8 further
            const float4 g4 = load4(xr + 16 * (c >> 3) + (c & 7), xvec), u4 = load4(xr + 16 * (c >> 3) + 8 + (c & 7), xvec);
            float4 v;
            v.x = __fmul_rn(__fdiv_rn(g4.x, __fadd_rn(1.0f, expf(-g4.x))), u4.x);
            v.y = __fmul_rn(__fdiv_rn(g4.y, __fadd_rn(1.0f, expf(-g4.y))), u4.y);
            v.z = __fmul_rn(__fdiv_rn(g4.z, __fadd_rn(1.0f, expf(-g4.z))), u4.z);
            v.w = __fmul_rn(__fdiv_rn(g4.w, __fadd_rn(1.0f, expf(-g4.w))), u4.w);
            *reinterpret_cast<float4*>(row + 4 * gi) = v;
            amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
    } else {
        for (int gi = threadIdx.x; gi < groups; gi += blockDim.x) {
            const float4 v = load4(xr + 4 * gi, xvec);
            *reinterpret_cast<float4*>(row + 4 * gi) = v;
            amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
    }
    amax = block_max<false>(amax, red_f);
    if (amax_out) {
        for (int gi = threadIdx.x; gi < groups; gi += blockDim.x)
            *reinterpret_cast<float4*>(v_out + (int64_t)b * k + 4 * gi) = *reinterpret_cast<const float4*>(row + 4 * gi);
        if (threadIdx.x == 0) amax_out[b] = __float_as_uint(amax);
        return;
    }
    if (amax_in) amax = __uint_as_float(amax_in[b]);
    const float s = __fdiv_rn(amax, 127.0f);
    const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    int local = 0;
    uint8_t* stage = reinterpret_cast<uint8_t*>(row + k);
    int8_t* qr = q ? q + (int64_t)b * q_stride : nullptr;
    const int groups_pad = qtc ? k_tiles * (kTileK / 4) : (int)(q_stride >> 2);
    for (int gi = threadIdx.x; gi < groups_pad; gi += blockDim.x) {
        int v[4] = {0, 0, 0, 0};
        if (gi < groups && amax > 0.0f) {
            const float4 f = *reinterpret_cast<const float4*>(row + 4 * gi);  // this thread's own values again
            v[0] = max(-127, min(127, ptx::round_half_away(__fmul_rn(f.x, inv))));
            v[1] = max(-127, min(127, ptx::round_half_away(__fmul_rn(f.y, inv))));
            v[2] = max(-127, min(127, ptx::round_half_away(__fmul_rn(f.z, inv))));
            v[3] = max(-127, min(127, ptx::round_half_away(__fmul_rn(f.w, inv))));
        }
        local += v[0] + v[1] + v[2] + v[3];
        if (qtc) {
            // residue r of k' = gi % 64 in k-tile gi / 64: staged at [k-tile][residue][k']
            const int kt = gi >> 6, kp = gi & 63;
#pragma unroll
            for (int r = 0; r < 4; ++r) stage[(kt * 4 + r) * 64 + kp] = (uint8_t)v[r];
        }
        if (qr)
            *reinterpret_cast<uint32_t*>(qr + 4 * gi) = (uint32_t)(v[0] & 0xff) | ((uint32_t)(v[1] & 0xff) << 8) |
                                                        ((uint32_t)(v[2] & 0xff) << 16) | ((uint32_t)(v[3] & 0xff) << 24);
    }
    if (v_out)
        for (int gi = threadIdx.x; gi < groups; gi += blockDim.x)
            *reinterpret_cast<float4*>(v_out + (int64_t)b * k + 4 * gi) = *reinterpret_cast<const float4*>(row + 4 * gi);
    const int total = block_sum_i(local, red_i);  // (its barriers also complete the staged bytes)
    if (qtc) {
        // 16-byte pieces [k-tile][residue][k' / 16] -> their places in the token block (gemm_tc_act_offset)
        const int tb = b / tc_nt, tin = b % tc_nt;
        int8_t* blk = qtc + (int64_t)tb * k_tiles * (4 * tc_nt * 64) + tin * 64;
        for (int pid = threadIdx.x; pid < k_tiles * 16; pid += blockDim.x) {
            const int kc = pid & 3, kr = pid >> 2;  // kr = k-tile * 4 + residue
            *reinterpret_cast<uint4*>(blk + (int64_t)kr * (tc_nt * 64) + ((kc ^ ((tin >> 1) & 3)) << 4)) = *reinterpret_cast<const uint4*>(stage + pid * 16);
        }
    }
    if (threadIdx.x == 0) {
        s_out[b] = s;
        qsum_out[b] = total;
    }
}

// The same row transform and quantiser into the tensor-core layout for many rows: a thread keeps its V groups of four
// values in registers from the load to the quantised bytes, all V loads in flight at once.  Bound by HBM and, for SiLU,
// by the instructions of the exponential and the exact divisions.  The kernel above holds a row in shared memory under
// 1024 threads: two rows per SM, each waiting for its loads and its barriers in turn.  A CTA of k / (4 V) threads leaves
// room for several rows per SM, so that one row's barriers hide under another's loads.  The bytes of a 4 x 4 block
// (four k' of a residue in a word, see gemm_tc_act_offset) are turned between four neighbouring lanes and go to global
// memory directly.
// Per launch before -> after (us): 2048 x 4096 RMSNorm 54.8 -> 17.8, identity 27.3 -> 10.5; 2048 x 14336 SiLU 82.2 -> 70.9
// (264 MB: 3.7 TB/s); 2001 x 14336 bf16 56.8 -> 39.7; 2044 x 2048 RMSNorm 21.1 -> 10.6; 64 x 4096 RMSNorm 4.9 -> 4.3.
// What is left is the instructions of the rounding: integers by one addition towards zero, without clamps, and their sum by dp4a
// took 2001 x 14336 bf16 from 41.2 to 34.9 and 2048 x 4096 RMSNorm from 17.9 to 16.4.
template <int PRE, typename T, int V>
__global__ void __launch_bounds__(512, V == 8 ? 2 : 3)
row_quant_many_kernel(const T* __restrict__ x, int64_t x_stride, const float* __restrict__ w, float eps, int k,
                      float* __restrict__ s_out, int32_t* __restrict__ qsum_out, int8_t* __restrict__ qtc, int tc_nt, int k_tiles) {
    __shared__ float red_f[32];
    __shared__ double red_d[32];
    __shared__ int red_i[32];
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const int b = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
    const T* xr = x + (int64_t)b * x_stride;
    const int groups = k >> 2, groups_pad = k_tiles * (kTileK / 4);
    float4 v[V];
    float amax = 0.0f;
    // (one decision on the alignment for all loads: a branch around each of them would let only one be in flight)
    auto load = [&](auto vec) {
        constexpr bool kVec = decltype(vec)::value;
        if constexpr (PRE == PRE_SWIGLU) {
            constexpr int kBatch = V < 4 ? V : 4;  // gate and up of four groups in flight
#pragma unroll
            for (int j0 = 0; j0 < V; j0 += kBatch) {
                float4 g[kBatch], u[kBatch];
#pragma unroll
                for (int j = 0; j < kBatch; ++j) {
                    const int c = 4 * (tid + (j0 + j) * nthr);  // outputs c .. c + 3: gate at x[16 (c / 8) + c % 8 ..], up 8 further
                    g[j] = u[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (c < k) {
                        g[j] = load4(xr + 16 * (c >> 3) + (c & 7), kVec);
                        u[j] = load4(xr + 16 * (c >> 3) + 8 + (c & 7), kVec);
                    }
                }
#pragma unroll
                for (int j = 0; j < kBatch; ++j) {
                    v[j0 + j].x = __fmul_rn(__fdiv_rn(g[j].x, __fadd_rn(1.0f, expf(-g[j].x))), u[j].x);
                    v[j0 + j].y = __fmul_rn(__fdiv_rn(g[j].y, __fadd_rn(1.0f, expf(-g[j].y))), u[j].y);
                    v[j0 + j].z = __fmul_rn(__fdiv_rn(g[j].z, __fadd_rn(1.0f, expf(-g[j].z))), u[j].z);
                    v[j0 + j].w = __fmul_rn(__fdiv_rn(g[j].w, __fadd_rn(1.0f, expf(-g[j].w))), u[j].w);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < V; ++j) {
                const int gi = tid + j * nthr;
                v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (gi < groups) v[j] = load4(xr + 4 * gi, kVec);
            }
        }
    };
    if ((reinterpret_cast<uintptr_t>(xr) & 15) == 0) load(std::true_type{});
    else load(std::false_type{});
    if (PRE == PRE_RMSNORM) {
        const bool wvec = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
        double ss = 0.0;  // f64, rounded once: reproducible against the CPU restatement
#pragma unroll
        for (int j = 0; j < V; ++j) {
            ss = fma((double)v[j].x, (double)v[j].x, ss);
            ss = fma((double)v[j].y, (double)v[j].y, ss);
            ss = fma((double)v[j].z, (double)v[j].z, ss);
            ss = fma((double)v[j].w, (double)v[j].w, ss);
        }
        ss = block_sum_d<false>(ss, red_d);
        const float denom = sqrtf(__fadd_rn((float)(ss / (double)k), eps));
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int gi = tid + j * nthr;
            if (gi < groups) {
                const float4 ww = load4(w + 4 * gi, wvec);
                v[j].x = __fmul_rn(__fdiv_rn(v[j].x, denom), ww.x);
                v[j].y = __fmul_rn(__fdiv_rn(v[j].y, denom), ww.y);
                v[j].z = __fmul_rn(__fdiv_rn(v[j].z, denom), ww.z);
                v[j].w = __fmul_rn(__fdiv_rn(v[j].w, denom), ww.w);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v[j].x), fabsf(v[j].y))), fmaxf(fabsf(v[j].z), fabsf(v[j].w)));
    amax = block_max<false>(amax, red_f);
    const float s = __fdiv_rn(amax, 127.0f);
    const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    int local = 0;
    // |v * inv| is 127 at most, up to two roundings, so that its integer needs no clamp; only where 127 / max|v| overflows it does
    const bool clamp = inv > 3.0e38f;
    const int lane = tid & 31, tin = b % tc_nt;
    int8_t* blk = qtc + (int64_t)(b / tc_nt) * k_tiles * (4 * tc_nt * 64) + (lane & 3) * (tc_nt * 64) + tin * 64;
    const uint32_t turn1 = lane & 1 ? 0x3715u : 0x6240u, turn2 = lane & 2 ? 0x3276u : 0x5410u;
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const int gi = tid + j * nthr;
        if (gi >= groups_pad) break;  // whole warps: groups_pad is a multiple of 64
        // (zeros behind the row, and all values of a row of zeros, whose inv is 0)
        int q[4] = {ptx::round_half_away(__fmul_rn(v[j].x, inv)), ptx::round_half_away(__fmul_rn(v[j].y, inv)),
                    ptx::round_half_away(__fmul_rn(v[j].z, inv)), ptx::round_half_away(__fmul_rn(v[j].w, inv))};
        if (clamp) {
#pragma unroll
            for (int e = 0; e < 4; ++e) q[e] = max(-127, min(127, q[e]));
        }
        // this lane has the residues 0 .. 3 of one k'; afterwards residue lane % 4 of four k'
        const uint32_t own = ptx::pack4_sat_s8(q[0], q[1], q[2], q[3]);
        local = ptx::dp4a_s8s8(own, 0x01010101u, local);
        const uint32_t half = __byte_perm(own, __shfl_xor_sync(0xffffffffu, own, 1), turn1);
        const uint32_t word = __byte_perm(half, __shfl_xor_sync(0xffffffffu, half, 2), turn2);
        const int kp = gi & 60;
        *reinterpret_cast<uint32_t*>(blk + (int64_t)(gi >> 6) * (4 * tc_nt * 64) + (((kp >> 4) ^ ((tin >> 1) & 3)) << 4) + (kp & 15)) = word;
    }
    const int total = block_sum_i(local, red_i);
    if (tid == 0) {
        s_out[b] = s;
        qsum_out[b] = total;
    }
}

// Greedy pick: the LAST index among equal maxima, as Iterator::max_by does in the
// reference's sampler (model/llama.rs:510-515).  One CTA per token.
__global__ void __launch_bounds__(1024) argmax_kernel(const float* __restrict__ logits, int64_t stride,
                                                      int vocab, int32_t* __restrict__ out) {
    __shared__ float sv[32];
    __shared__ int si[32];
    ptx::pdl_wait();
    const float* row = logits + (int64_t)blockIdx.x * stride;
    float best = -INFINITY;
    int idx = -1;
    if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
        // four consecutive values per load, four loads in flight per thread; within a thread the indices rise,
        // so ">=" keeps the last of equal maxima
        const int groups = vocab >> 2;
        for (int g0 = threadIdx.x; g0 < groups; g0 += 4 * blockDim.x) {
            float4 f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int gi = g0 + u * blockDim.x;
                f[u] = gi < groups ? *reinterpret_cast<const float4*>(row + 4 * gi) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = 4 * (g0 + u * blockDim.x);
                if (c < 4 * groups) {
                    if (f[u].x >= best || idx < 0) { best = f[u].x; idx = c; }
                    if (f[u].y >= best) { best = f[u].y; idx = c + 1; }
                    if (f[u].z >= best) { best = f[u].z; idx = c + 2; }
                    if (f[u].w >= best) { best = f[u].w; idx = c + 3; }
                }
            }
        }
        for (int c = 4 * groups + threadIdx.x; c < vocab; c += blockDim.x) {
            const float v = row[c];
            if (v >= best || idx < 0) { best = v; idx = c; }
        }
    } else {
        for (int c = threadIdx.x; c < vocab; c += blockDim.x) {
            const float v = row[c];
            if (v >= best || idx < 0) { best = v; idx = c; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (oi >= 0 && (idx < 0 || ov > best || (ov == best && oi > idx))) { best = ov; idx = oi; }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sv[w] = best; si[w] = idx; }
    __syncthreads();
    if (w == 0) {
        best = l < (blockDim.x >> 5) ? sv[l] : -INFINITY;
        idx = l < (blockDim.x >> 5) ? si[l] : -1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (oi >= 0 && (idx < 0 || ov > best || (ov == best && oi > idx))) { best = ov; idx = oi; }
        }
        if (l == 0) out[blockIdx.x] = idx;
    }
}


// Dense lm_head (candle_nn::Linear without bias, model/llama.rs:23,266; the converter keeps it in 16 bits,
// tools/conversion/convert_llama_v2.py:265-268) with the final RMSNorm folded in (every CTA normalises the
// hidden vector itself, sum of squares in f64) and a running arg-max per CTA, so that the greedy pick does
// not need a pass over all logits.  Ties keep the larger index (model/llama.rs:510-515).  HBM-bound on W:
// one warp per output row, 16-byte loads, x in shared memory, f32 accumulation.
// PAD: rows of w (and xs) are `ld_pad` apart instead of `hidden`.
template <int B, bool F16, bool PAD>
__global__ void __launch_bounds__(256) lm_head_fused_kernel(const __nv_bfloat16* __restrict__ w,
                                                            const float* __restrict__ h,
                                                            const float* __restrict__ norm_w, float eps,
                                                            int hidden, int ld_pad, int64_t vocab, float* __restrict__ logits,
                                                            float* __restrict__ cand_val,
                                                            int32_t* __restrict__ cand_idx, float cap) {
    const int ld = PAD ? ld_pad : hidden;
    extern __shared__ float xs[];  // [B][ld], zero beyond hidden
    __shared__ double red_d[32];
    __shared__ float best_v[8][B];
    __shared__ int best_i[8][B];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t warp_global = (int64_t)blockIdx.x * 8 + warp;
    const int64_t warps_total = (int64_t)gridDim.x * 8;
    // One token: the weights stream through two sets of registers, across the ends of rows.  kBatch chunks of 16 bytes per
    // lane are on their way while the set before is multiplied, the first ones before the wait for the kernel in front
    // (they depend on nothing).  Without that a warp asks for four chunks when it has used up the last four, and for a
    // row's first after the reduction of the row before: 32000 x 4096 77.9 -> 63.4 us (4.1 TB/s), 32000 x 2048 43.7 -> 35.2.
    // With more tokens the second set costs resident CTAs (two tokens 130 -> 137 us, four 176 -> 235): they keep the loop.
    constexpr bool kAhead = B == 1;
    constexpr int kBatch = kAhead ? 4 : 1;
    const int n8 = ld / 8;
    int64_t next_v = warp_global;
    int next_c = 0;
    uint4 ahead[kBatch];
    auto load = [&]() {  // the next batch
        const uint4* wr = reinterpret_cast<const uint4*>(w + next_v * ld);
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int c8 = next_c + 32 * u + lane;
            ahead[u] = make_uint4(0u, 0u, 0u, 0u);
            if (next_v < vocab && c8 < n8) ahead[u] = __ldg(wr + c8);
        }
        next_c += 32 * kBatch;
        if (next_c >= n8) { next_c = 0; next_v += warps_total; }
    };
    if (kAhead) load();
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    for (int b = 0; b < B; ++b) {
        double ss = 0.0;
        for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
            const float v = h[(int64_t)b * hidden + c];
            xs[b * ld + c] = v;
            ss = fma((double)v, (double)v, ss);
        }
        ss = block_sum_d(ss, red_d);
        const float denom = sqrtf(__fadd_rn((float)(ss / (double)hidden), eps));
        for (int c = threadIdx.x; c < hidden; c += blockDim.x)
            xs[b * ld + c] = __fmul_rn(__fdiv_rn(xs[b * ld + c], denom), norm_w[c]);
        if (PAD)
            for (int c = hidden + threadIdx.x; c < ld; c += blockDim.x) xs[b * ld + c] = 0.0f;
    }
    __syncthreads();
    float bv[B];
    int bi[B];
#pragma unroll
    for (int b = 0; b < B; ++b) { bv[b] = -INFINITY; bi[b] = -1; }
    for (int64_t v = warp_global; v < vocab; v += warps_total) {
        float acc[B];
#pragma unroll
        for (int b = 0; b < B; ++b) acc[b] = 0.0f;
        auto multiply = [&](const uint4& pk, int c8) {
            const uint32_t u[4] = {pk.x, pk.y, pk.z, pk.w};
            float wf[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack16<F16>(u[j], wf[2 * j], wf[2 * j + 1]);
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const float4 x0 = *reinterpret_cast<const float4*>(xs + b * ld + c8 * 8);
                const float4 x1 = *reinterpret_cast<const float4*>(xs + b * ld + c8 * 8 + 4);
                acc[b] = fmaf(wf[0], x0.x, acc[b]);
                acc[b] = fmaf(wf[1], x0.y, acc[b]);
                acc[b] = fmaf(wf[2], x0.z, acc[b]);
                acc[b] = fmaf(wf[3], x0.w, acc[b]);
                acc[b] = fmaf(wf[4], x1.x, acc[b]);
                acc[b] = fmaf(wf[5], x1.y, acc[b]);
                acc[b] = fmaf(wf[6], x1.z, acc[b]);
                acc[b] = fmaf(wf[7], x1.w, acc[b]);
            }
        };
        if constexpr (kAhead) {
            for (int c = 0; c < n8; c += 32 * kBatch) {
                uint4 now[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) now[i] = ahead[i];
                load();
#pragma unroll
                for (int i = 0; i < kBatch; ++i)
                    if (c + 32 * i + lane < n8) multiply(now[i], c + 32 * i + lane);
            }
        } else {
            const uint4* wr = reinterpret_cast<const uint4*>(w + v * ld);
#pragma unroll 4
            for (int c8 = lane; c8 < n8; c8 += 32) multiply(wr[c8], c8);
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            float r = warp_sum(acc[b]);
            if (PAD && cap > 0.0f) r = cap * tanhf(r / cap);
            if (lane == 0) logits[(int64_t)b * vocab + v] = r;
            if (r >= bv[b]) { bv[b] = r; bi[b] = (int)v; }  // v increases: ties keep the later index
        }
    }
    if (lane == 0)
#pragma unroll
        for (int b = 0; b < B; ++b) { best_v[warp][b] = bv[b]; best_i[warp][b] = bi[b]; }
    __syncthreads();
    if (threadIdx.x < B) {
        const int b = threadIdx.x;
        float v = -INFINITY;
        int i = -1;
        for (int wv = 0; wv < 8; ++wv) {
            const float ov = best_v[wv][b];
            const int oi = best_i[wv][b];
            if (oi >= 0 && (i < 0 || ov > v || (ov == v && oi > i))) { v = ov; i = oi; }
        }
        cand_val[(int64_t)b * gridDim.x + blockIdx.x] = v;
        cand_idx[(int64_t)b * gridDim.x + blockIdx.x] = i;
    }
}

// The same for one token, rows of a multiple of 256 values: every warp owns a run of neighbouring rows, a stream of bytes that it
// brings into its own ring in shared memory with bulk copies, kHeadSlot bytes at a time, so that 192 KB an SM are on their way
// whatever the warps do; the first ones are requested before the wait for the kernel in front.  Through registers (above) 64 KB
// an SM were.  Bound by the reads of the weights: 32000 x 4096 64 -> 57 us, 4.6 TB/s (the same with slots of 2 KB, six a warp; 64 with
// eight warps and slots of 8 KB).  Sums in the same order.  Rows of other lengths, or more than 8192 values, stay with the kernel
// above; so do several tokens, whose values for one row the rings leave no room for.
constexpr int kHeadWarps = 16, kHeadSlot = 4096, kHeadSlots = 3, kHeadMaxLd = 8192;
constexpr unsigned kErrHeadTimeout = 0x48454144u;  // 'HEAD'
template <bool F16>
__global__ void __launch_bounds__(kHeadWarps * 32, 1) lm_head_stream_kernel(const __nv_bfloat16* __restrict__ w, const float* __restrict__ h, const float* __restrict__ norm_w,
                                                                            float eps, int hidden, int ld, int64_t vocab, float* __restrict__ logits, float* __restrict__ cand_val,
                                                                            int32_t* __restrict__ cand_idx, float cap, unsigned int* err) {
    extern __shared__ __align__(128) uint8_t hsm[];  // rings | x
    __shared__ uint64_t full[kHeadWarps][kHeadSlots];
    __shared__ double red_d[32];
    __shared__ float best_v[kHeadWarps];
    __shared__ int best_i[kHeadWarps];
    float* xs = reinterpret_cast<float*>(hsm + kHeadWarps * kHeadSlots * kHeadSlot);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t wg = (int64_t)blockIdx.x * kHeadWarps + warp, warps = (int64_t)gridDim.x * kHeadWarps;
    const int64_t v0 = vocab * wg / warps, v1 = vocab * (wg + 1) / warps;
    uint8_t* ring = hsm + warp * (kHeadSlots * kHeadSlot);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(w + v0 * ld);
    const int64_t bytes = (v1 - v0) * ld * 2;
    const int slots = (int)((bytes + kHeadSlot - 1) / kHeadSlot);
    auto request = [&](int i) {  // lane 0
        const int64_t left = bytes - (int64_t)i * kHeadSlot;
        const uint32_t n = (uint32_t)(left < kHeadSlot ? left : kHeadSlot);
        ptx::mbar_arrive_expect_tx(&full[warp][i % kHeadSlots], n);
        ptx::bulk_g2s(ring + (i % kHeadSlots) * kHeadSlot, src + (int64_t)i * kHeadSlot, n, &full[warp][i % kHeadSlots]);
    };
    if (lane < kHeadSlots) ptx::mbar_init(&full[warp][lane], 1);
    ptx::mbar_fence_init();
    __syncwarp();
    if (lane == 0)
        for (int i = 0; i < kHeadSlots && i < slots; ++i) request(i);
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    double ss = 0.0;
    for (int c = threadIdx.x; c < hidden; c += blockDim.x) {
        const float v = h[c];
        xs[c] = v;
        ss = fma((double)v, (double)v, ss);
    }
    ss = block_sum_d(ss, red_d);
    const float denom = sqrtf(__fadd_rn((float)(ss / (double)hidden), eps));
    for (int c = threadIdx.x; c < ld; c += blockDim.x) xs[c] = c < hidden ? __fmul_rn(__fdiv_rn(xs[c], denom), norm_w[c]) : 0.0f;
    __syncthreads();
    float bv = -INFINITY, acc = 0.0f;
    int bi = -1, c8 = lane;
    const int n8 = ld / 8;  // pieces of 16 bytes to a row, a multiple of 32
    int64_t v = v0;
    bool ok = true;
    for (int i = 0; i < slots; ++i) {
        ok &= ptx::mbar_wait_bounded(&full[warp][i % kHeadSlots], (uint32_t)((i / kHeadSlots) & 1));
        const uint4* at = reinterpret_cast<const uint4*>(ring + (i % kHeadSlots) * kHeadSlot) + lane;
#pragma unroll 4
        for (int u = 0; u < kHeadSlot / 512; ++u) {
            const uint4 now = at[32 * u];  // (the last slot's end may hold older bytes: not used)
            if (v >= v1) break;
            const uint32_t p[4] = {now.x, now.y, now.z, now.w};
            const float4 x0 = *reinterpret_cast<const float4*>(xs + c8 * 8), x1 = *reinterpret_cast<const float4*>(xs + c8 * 8 + 4);
            float wf[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) unpack16<F16>(p[j], wf[2 * j], wf[2 * j + 1]);
            acc = fmaf(wf[0], x0.x, acc);
            acc = fmaf(wf[1], x0.y, acc);
            acc = fmaf(wf[2], x0.z, acc);
            acc = fmaf(wf[3], x0.w, acc);
            acc = fmaf(wf[4], x1.x, acc);
            acc = fmaf(wf[5], x1.y, acc);
            acc = fmaf(wf[6], x1.z, acc);
            acc = fmaf(wf[7], x1.w, acc);
            c8 += 32;
            if (c8 >= n8) {
                float r = warp_sum(acc);
                if (cap > 0.0f) r = cap * tanhf(r / cap);
                if (lane == 0) logits[v] = r;
                if (r >= bv) { bv = r; bi = (int)v; }  // v increases: ties keep the later index
                acc = 0.0f;
                c8 = lane;
                ++v;
            }
        }
        __syncwarp();  // the slot has been read
        if (lane == 0 && i + kHeadSlots < slots) request(i + kHeadSlots);
    }
    if (!ok && lane == 0) {
        atomicExch(err, kErrHeadTimeout);
        // copies still in flight get a bounded chance to land before the CTA retires
        for (int k = 0; k < kHeadSlots && k < slots; ++k) ptx::mbar_wait_bounded(&full[warp][k], (uint32_t)(((slots - 1 - k) / kHeadSlots) & 1), 1u << 16);
    }
    if (lane == 0) { best_v[warp] = bv; best_i[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = -INFINITY;
        int at = -1;
        for (int k = 0; k < kHeadWarps; ++k)
            if (best_i[k] >= 0 && (at < 0 || best_v[k] > b || (best_v[k] == b && best_i[k] > at))) { b = best_v[k]; at = best_i[k]; }
        cand_val[blockIdx.x] = b;
        cand_idx[blockIdx.x] = at;
    }
}

__global__ void __launch_bounds__(256) pick_kernel(const float* __restrict__ cand_val,
                                                   const int32_t* __restrict__ cand_idx, int n_cand,
                                                   int32_t* __restrict__ out, int32_t* __restrict__ pos, int n_pos) {
    __shared__ float sv[8];
    __shared__ int si[8];
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const int b = blockIdx.x;
    float v = -INFINITY;
    int i = -1;
    for (int c = threadIdx.x; c < n_cand; c += blockDim.x) {
        const float ov = cand_val[(int64_t)b * n_cand + c];
        const int oi = cand_idx[(int64_t)b * n_cand + c];
        if (oi >= 0 && (i < 0 || ov > v || (ov == v && oi > i))) { v = ov; i = oi; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (oi >= 0 && (i < 0 || ov > v || (ov == v && oi > i))) { v = ov; i = oi; }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { sv[w] = v; si[w] = i; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) {
            const float ov = sv[k];
            const int oi = si[k];
            if (oi >= 0 && (i < 0 || ov > v || (ov == v && oi > i))) { v = ov; i = oi; }
        }
        out[b] = i;
    }
    if (b == 0 && threadIdx.x < n_pos) pos[threadIdx.x] += 1;  // BitLlama::current_pos += 1, model/llama.rs:269
}

// h += y over n floats (the residual add after a projection whose bases were summed into y first)
__global__ void __launch_bounds__(256) residual_add_kernel(float* __restrict__ h, const float* __restrict__ y, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        h[i] = __fadd_rn(h[i], y[i]);
}

}  // namespace

cudaError_t launch_residual_add(float* h, const float* y, int64_t n, cudaStream_t stream) {
    const int64_t blocks = (n + 255) / 256;
    residual_add_kernel<<<(unsigned)(blocks < 1184 ? blocks : 1184), 256, 0, stream>>>(h, y, n);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
cudaError_t launch_embed(const int32_t* tokens, const __nv_bfloat16* table, int batch, int hidden,
                         int vocab, float* h, cudaStream_t stream, unsigned int* clear, int n_clear, bool pdl, bool f16) {
    return launch_pdl(embed_kernel, dim3(batch), dim3(256), 0, stream, pdl, tokens, table, hidden, vocab, h, clear,
                      n_clear, f16);
}

// Rows that the kernel takes: the values and, for the tensor-core product, their bytes in shared memory.
bool row_quant_fits(int64_t k, int64_t k_tiles) { return 4 * k + k_tiles * kTileK <= 200 * 1024; }

// The kernel that keeps its values in registers: 2 groups of four values a thread while a row's own latency counts, 8 groups
// beyond that, where several rows share an SM in turn (2044 x 2048 RMSNorm: 12.2 us with 2 groups, 10.6 with 8; 64 x 4096:
// 4.3 and 7.7).  The line between them is a measured one, for the 148 SMs of a B200: 2048 threads of 2 groups a SM (of which
// 1536 can be resident: 32 to 35 registers, 512 threads a CTA).  Few rows too wide for 512 threads of 2 groups stay with
// the kernel above (64 rows x 14336, SiLU: 6.8 us there, 7.3 us with 8 groups a thread).
static constexpr int64_t kFewRowGroups = 2ll * 148 * 2048;
static int row_quant_groups(int batch, int groups) {  // groups per thread; 0: the kernel above
    if ((int64_t)batch * groups <= kFewRowGroups) return groups <= 2 * 512 ? 2 : (batch >= 256 && groups <= 8 * 512 ? 8 : 0);
    return groups <= 8 * 512 ? 8 : 0;
}

template <int PRE, typename T>
static cudaError_t launch_row_quant_many(const T* x, int64_t x_stride, const float* w, float eps, int batch, int k, float* s, int32_t* qsum,
                                         cudaStream_t stream, int8_t* qtc, int tc_nt, int k_tiles) {
    const int groups = k_tiles * (kTileK / 4), per = row_quant_groups(batch, groups);
    const dim3 grid((unsigned)batch), block((unsigned)((groups + 32 * per - 1) / (32 * per) * 32));
    if (per == 8)
        return launch_pdl(row_quant_many_kernel<PRE, T, 8>, grid, block, 0, stream, false, x, x_stride, w, eps, k, s, qsum, qtc, tc_nt, k_tiles);
    return launch_pdl(row_quant_many_kernel<PRE, T, 2>, grid, block, 0, stream, false, x, x_stride, w, eps, k, s, qsum, qtc, tc_nt, k_tiles);
}

cudaError_t launch_row_quant(int pre, const float* x, int64_t x_stride, const float* w, float eps,
                             int batch, int k, int8_t* q, int64_t q_stride, float* s, int32_t* qsum,
                             float* v_out, cudaStream_t stream, int8_t* qtc, int k_tiles,
                             const unsigned int* amax_in, unsigned int* amax_out) {
    const int tc_nt = batch <= 64 ? 64 : 128;
    if (amax_out && !v_out) return cudaErrorInvalidValue;
    if (k % 4 != 0 || (q && q_stride % 4 != 0)) return cudaErrorInvalidValue;
    if (qtc && !q && !v_out && !amax_in && !amax_out && row_quant_groups(batch, k_tiles * (kTileK / 4)) > 0) {
        if (pre == PRE_RMSNORM) return launch_row_quant_many<PRE_RMSNORM>(x, x_stride, w, eps, batch, k, s, qsum, stream, qtc, tc_nt, k_tiles);
        if (pre == PRE_SWIGLU) return launch_row_quant_many<PRE_SWIGLU>(x, x_stride, w, eps, batch, k, s, qsum, stream, qtc, tc_nt, k_tiles);
        return launch_row_quant_many<PRE_NONE>(x, x_stride, w, eps, batch, k, s, qsum, stream, qtc, tc_nt, k_tiles);
    }
    const size_t smem = (size_t)k * sizeof(float) + (qtc ? (size_t)k_tiles * kTileK : 0);
    const int threads = k >= 4096 ? 1024 : (k >= 2048 ? 512 : 256);
    static PerDeviceOnce once;
    cudaError_t ce = once.run([] {
        cudaError_t e = cudaFuncSetAttribute(row_quant_kernel<PRE_NONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(row_quant_kernel<PRE_RMSNORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(row_quant_kernel<PRE_SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        return e;
    });
    if (ce != cudaSuccess) return ce;
    if (smem > 200 * 1024) return cudaErrorInvalidConfiguration;
    // an ordinary launch (starting early behind a tensor-core product measured slower inside the decode step); the
    // kernel still releases its own dependent at once, so that the product behind it can fetch weights meanwhile
    const dim3 grid((unsigned)batch), block((unsigned)threads);
    if (pre == PRE_RMSNORM)
        return launch_pdl(row_quant_kernel<PRE_RMSNORM>, grid, block, smem, stream, false, x, x_stride, w, eps, k, q, q_stride, s, qsum, v_out, qtc, tc_nt, k_tiles, amax_in, amax_out);
    if (pre == PRE_SWIGLU)
        return launch_pdl(row_quant_kernel<PRE_SWIGLU>, grid, block, smem, stream, false, x, x_stride, w, eps, k, q, q_stride, s, qsum, v_out, qtc, tc_nt, k_tiles, amax_in, amax_out);
    return launch_pdl(row_quant_kernel<PRE_NONE>, grid, block, smem, stream, false, x, x_stride, w, eps, k, q, q_stride, s, qsum, v_out, qtc, tc_nt, k_tiles, amax_in, amax_out);
}

// Identity transform + quantiser on bf16 rows, into the tensor-core product's layout.
cudaError_t launch_row_quant_bf16(const __nv_bfloat16* x, int64_t x_stride, int batch, int k, float* s, int32_t* qsum,
                                  cudaStream_t stream, int8_t* qtc, int k_tiles) {
    const int tc_nt = batch <= 64 ? 64 : 128;
    if (k % 4 != 0 || !qtc) return cudaErrorInvalidValue;
    if (row_quant_groups(batch, k_tiles * (kTileK / 4)) > 0)
        return launch_row_quant_many<PRE_NONE>(x, x_stride, nullptr, 0.0f, batch, k, s, qsum, stream, qtc, tc_nt, k_tiles);
    const size_t smem = (size_t)k * sizeof(float) + (size_t)k_tiles * kTileK;
    const int threads = k >= 4096 ? 1024 : (k >= 2048 ? 512 : 256);
    static PerDeviceOnce once;
    cudaError_t ce = once.run([] { return cudaFuncSetAttribute(row_quant_kernel<PRE_NONE, __nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
    if (ce != cudaSuccess) return ce;
    if (smem > 200 * 1024) return cudaErrorInvalidConfiguration;
    return launch_pdl(row_quant_kernel<PRE_NONE, __nv_bfloat16>, dim3((unsigned)batch), dim3((unsigned)threads), smem, stream, false, x, x_stride,
                      (const float*)nullptr, 0.0f, k, (int8_t*)nullptr, (int64_t)0, s, qsum, (float*)nullptr, qtc, tc_nt, k_tiles,
                      (const unsigned int*)nullptr, (unsigned int*)nullptr);
}

cudaError_t launch_argmax(const float* logits, int batch, int vocab, int32_t* out, cudaStream_t stream) {
    argmax_kernel<<<batch, 1024, 0, stream>>>(logits, vocab, vocab, out);
    return cudaGetLastError();
}

int lm_head_max_candidates(int sm_count) { return sm_count * 4; }

template <int B, bool F16, bool PAD>
static cudaError_t launch_lm_head_fused_bt(const __nv_bfloat16* w, const float* h, const float* norm_w, float eps,
                                           int hidden, int ld, int64_t vocab, float* logits, float* cand_val,
                                           int32_t* cand_idx, int grid, cudaStream_t stream, bool pdl, float cap) {
    const size_t smem = (size_t)B * ld * sizeof(float);
    static PerDeviceOnce once;
    cudaError_t ce = once.run([] { return cudaFuncSetAttribute(lm_head_fused_kernel<B, F16, PAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
    if (ce != cudaSuccess) return ce;
    if (smem > 200 * 1024) return cudaErrorInvalidConfiguration;
    return launch_pdl(lm_head_fused_kernel<B, F16, PAD>, dim3(grid), dim3(256), smem, stream, pdl, w, h, norm_w, eps, hidden, ld,
                      vocab, logits, cand_val, cand_idx, cap);
}
template <int B>
static cudaError_t launch_lm_head_fused_b(const __nv_bfloat16* w, const float* h, const float* norm_w, float eps,
                                          int hidden, int ld, int64_t vocab, float* logits, float* cand_val,
                                          int32_t* cand_idx, int grid, cudaStream_t stream, bool pdl, bool f16, float cap) {
    if (ld != hidden || cap > 0.0f)  // bf16 tables only
        return f16 ? cudaErrorInvalidValue
                   : launch_lm_head_fused_bt<B, false, true>(w, h, norm_w, eps, hidden, ld, vocab, logits, cand_val, cand_idx, grid, stream, pdl, cap);
    return f16 ? launch_lm_head_fused_bt<B, true, false>(w, h, norm_w, eps, hidden, ld, vocab, logits, cand_val, cand_idx, grid, stream, pdl, cap)
               : launch_lm_head_fused_bt<B, false, false>(w, h, norm_w, eps, hidden, ld, vocab, logits, cand_val, cand_idx, grid, stream, pdl, cap);
}

cudaError_t launch_lm_head_fused(const __nv_bfloat16* w, const float* h, const float* norm_w, float eps,
                                 int batch, int hidden, int64_t vocab, float* logits, float* cand_val,
                                 int32_t* cand_idx, int* n_cand, int sm_count, cudaStream_t stream, bool pdl, bool f16, int ld, float cap) {
    if (ld == 0) ld = hidden;
    if (ld % 8 != 0 || ld < hidden || batch < 1) return cudaErrorInvalidValue;
    // (a row must be whole pieces of a warp: 32 lanes x 8 values)
    if (batch == 1 && ld % 256 == 0 && ld <= kHeadMaxLd && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && !(f16 && (ld != hidden || cap > 0.0f))) {
        constexpr size_t rings = (size_t)kHeadWarps * kHeadSlots * kHeadSlot;
        static PerDeviceOnce once;
        cudaError_t ce = once.run([] {
            cudaError_t e = cudaFuncSetAttribute(lm_head_stream_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(rings + kHeadMaxLd * sizeof(float)));
            return e == cudaSuccess ? cudaFuncSetAttribute(lm_head_stream_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(rings + kHeadMaxLd * sizeof(float))) : e;
        });
        int dev = 0;
        if (ce == cudaSuccess) ce = cudaGetDevice(&dev);
        if (ce != cudaSuccess) return ce;
        *n_cand = sm_count;
        return launch_pdl(f16 ? lm_head_stream_kernel<true> : lm_head_stream_kernel<false>, dim3((unsigned)sm_count), dim3(kHeadWarps * 32), rings + ld * sizeof(float), stream, pdl,
                          w, h, norm_w, eps, hidden, ld, vocab, logits, cand_val, cand_idx, cap, device_error_word(dev));
    }
    // one grid size for every group of tokens, so that the candidate rows share a stride
    const int per_pass = batch > 4 ? 8 : 4;  // tokens per pass over the weights
    const size_t smem_max = (size_t)(batch < per_pass ? batch : per_pass) * ld * sizeof(float);
    int per_sm = (int)((200 * 1024) / (smem_max + 2048));
    per_sm = per_sm > 4 ? 4 : (per_sm < 1 ? 1 : per_sm);
    const int grid = sm_count * per_sm;
    *n_cand = grid;
    for (int b0 = 0; b0 < batch; b0 += per_pass) {
        const int bc = batch - b0 < per_pass ? batch - b0 : per_pass;
        const float* hb = h + (size_t)b0 * hidden;
        float* lb = logits + (size_t)b0 * vocab;
        float* cv = cand_val + (size_t)b0 * grid;
        int32_t* ci = cand_idx + (size_t)b0 * grid;
        cudaError_t e;
        switch (bc) {
            case 1: e = launch_lm_head_fused_b<1>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            case 2: e = launch_lm_head_fused_b<2>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            case 3: e = launch_lm_head_fused_b<3>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            case 4: e = launch_lm_head_fused_b<4>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            case 5: e = launch_lm_head_fused_b<5>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            case 6: e = launch_lm_head_fused_b<6>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            case 7: e = launch_lm_head_fused_b<7>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
            default: e = launch_lm_head_fused_b<8>(w, hb, norm_w, eps, hidden, ld, vocab, lb, cv, ci, grid, stream, pdl, f16, cap); break;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_pick(const float* cand_val, const int32_t* cand_idx, int n_cand, int batch, int32_t* out,
                        int32_t* pos, int n_pos, cudaStream_t stream, bool pdl) {
    return launch_pdl(pick_kernel, dim3(batch), dim3(256), 0, stream, pdl, cand_val, cand_idx, n_cand, out, pos, n_pos);
}

}  // namespace bt

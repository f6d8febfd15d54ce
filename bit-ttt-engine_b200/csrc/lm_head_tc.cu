// Dense bf16 lm_head for more than 8 tokens on the tensor cores (tcgen05, kind::f16):
//   logits[m, v] = sum_c W[v, c] * xn[m, c],  xn = RMSNorm(h)   (model/llama.rs:256-266).
// W is bf16; xn is f32 and is split into two bf16 terms hi + lo (error ~2^-17 relative), which
// ride as 2 x 64 columns of one N = 128 product and are added in the epilogue, so the result
// stays within ~1e-5 of the f32 reference instead of the 4e-3 of a plain bf16 cast.
// W is kept in a second, tile-ordered copy (128 rows x 64 inputs per 16 KB tile, 8x16-byte core
// matrices, K-major, no swizzle) so that one 1-D bulk copy fetches an operand tile.
#include "bt_common.cuh"
#include "bt_model.cuh"
#include "bt_ptx.cuh"

namespace bt {

namespace {

constexpr int kRows = 128, kChunk = 64, kTok = 64, kCols = 2 * kTok;  // N = hi | lo
constexpr int kATile = kRows * kChunk * 2;                              // 16 KB
constexpr int kBTile = kCols * kChunk * 2;                              // 16 KB
// As many chunks of weights and activations in flight as fit: bound by the reads of the weights, and 16 tokens bring a quarter of
// the activations of 64, so that eleven stages fit instead of four (32000 x 2560, 16 tokens: 34 -> 29 us).
constexpr int kRingBytes = 224 * 1024, kMaxStages = 12;
constexpr int kThreads = 6 * 32;
constexpr unsigned kErrLmTimeout = 0x4c4d4844u;  // 'LMHD'

// kind::f16: D = f32, A (the weights) and B (the activation pieces) both bf16 or both IEEE half - the two
// operand formats of one instruction must be the same 16-bit type - K-major, M x N tile
__device__ __forceinline__ uint32_t instr_desc_bf16(int m, int n, bool f16) {
    uint32_t d = 0;
    d |= 1u << 4;                    // accumulator format: f32
    d |= (f16 ? 0u : 1u) << 7;       // A format: 0 = f16, 1 = bf16
    d |= (f16 ? 0u : 1u) << 10;      // B format
    d |= (uint32_t)(n >> 3) << 17;
    d |= (uint32_t)(m >> 4) << 24;
    return d;
}

// byte offset of element (row, c) inside a K-major tile with `chunk` 2-byte inputs per row
__device__ __host__ __forceinline__ int64_t tile_off(int row, int c, int chunk) {
    return (int64_t)(row >> 3) * (chunk / 8) * 128 + (c >> 3) * 128 + (row & 7) * 16 + (c & 7) * 2;
}

// row-major bf16 [vocab, hidden] -> tiles [row_set][k_chunk][16 KB]
__global__ void lm_retile_kernel(const __nv_bfloat16* __restrict__ w, int64_t vocab, int hidden, int ld,
                                 __nv_bfloat16* __restrict__ tiles) {
    const int64_t row_sets = (vocab + kRows - 1) / kRows;
    const int chunks = (hidden + kChunk - 1) / kChunk;
    const int64_t total = row_sets * chunks * (kRows * kChunk);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t tile = i / (kRows * kChunk);
        const int e = (int)(i % (kRows * kChunk));
        const int row = e / kChunk, c = e % kChunk;
        const int64_t rs = tile / chunks;
        const int kc = (int)(tile % chunks);
        const int64_t v = rs * kRows + row;
        const __nv_bfloat16 val = v < vocab && kc * kChunk + c < hidden ? w[v * ld + kc * kChunk + c] : __float2bfloat16_rn(0.0f);
        *reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<uint8_t*>(tiles) + tile * kATile + tile_off(row, c, kChunk)) = val;
    }
}

// RMSNorm of up to 64 tokens, split into bf16 hi | lo, laid out as the B tiles of every k-chunk
// f16: the pieces are IEEE halves (hi + lo = 11 + 11 significand bits; a lo piece below 6e-5 is subnormal and
// keeps an absolute accuracy of 2^-25) to match weights stored as halves; otherwise bf16 (8 + 8 bits).
// cols: columns of the product, hi | lo of cols / 2 tokens.  A thread takes eight inputs at a time (one 16-byte piece of either
// part), and up to kPrepKeep of them stay in registers between the two passes (64 x 4096: 12.5 us with a value a thread, 3 us).
constexpr int kPrepThreads = 256, kPrepKeep = 2;
__global__ void __launch_bounds__(kPrepThreads) lm_prep_kernel(const float* __restrict__ h, const float* __restrict__ norm_w,
                                                               float eps, int hidden, int m, int cols, uint8_t* __restrict__ btiles, bool f16) {
    __shared__ double red[32];
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const int token = blockIdx.x;  // 0 .. cols / 2 - 1
    const bool real = token < m;
    const float* hr = h + (int64_t)(real ? token : 0) * hidden;
    const bool vec = ((reinterpret_cast<uintptr_t>(hr) | reinterpret_cast<uintptr_t>(norm_w)) & 15) == 0;
    auto get = [&](const float* p, int c0, float (&v)[8]) {
        if (vec && c0 + 8 <= hidden) {
            const float4 x = *reinterpret_cast<const float4*>(p + c0), y = *reinterpret_cast<const float4*>(p + c0 + 4);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = c0 + j < hidden ? p[c0 + j] : 0.0f;
        }
    };
    const int padded = (hidden + kChunk - 1) / kChunk * kChunk;
    float keep[kPrepKeep][8];
    double ss = 0.0;
    auto squares = [&](const float (&v)[8]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fma((double)v[j], (double)v[j], ss);
    };
#pragma unroll
    for (int i = 0; i < kPrepKeep; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) keep[i][j] = 0.0f;
        if (real) get(hr, (i * kPrepThreads + (int)threadIdx.x) * 8, keep[i]);
        squares(keep[i]);
    }
    if (real)
        for (int c0 = (kPrepKeep * kPrepThreads + (int)threadIdx.x) * 8; c0 < hidden; c0 += kPrepThreads * 8) {
            float v[8];
            get(hr, c0, v);
            squares(v);
        }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.0;
    for (int w = 0; w < kPrepThreads / 32; ++w) ss += red[w];
    const float denom = sqrtf(__fadd_rn((float)(ss / (double)hidden), eps));
    auto put = [&](int c0, const float (&x)[8]) {
        if (c0 >= padded) return;
        float w[8];
        uint32_t hi[4], lo[4];
        get(norm_w, c0, w);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const float a = real ? __fmul_rn(__fdiv_rn(x[j], denom), w[j]) : 0.0f, b = real ? __fmul_rn(__fdiv_rn(x[j + 1], denom), w[j + 1]) : 0.0f;
            if (f16) {
                const __half2 u = __floats2half2_rn(a, b), l = __floats2half2_rn(a - __low2float(u), b - __high2float(u));
                hi[j / 2] = *reinterpret_cast<const uint32_t*>(&u);
                lo[j / 2] = *reinterpret_cast<const uint32_t*>(&l);
            } else {
                hi[j / 2] = ptx::pack2(a, b);
                lo[j / 2] = ptx::pack2(a - __uint_as_float(hi[j / 2] << 16), b - __uint_as_float(hi[j / 2] & 0xffff0000u));
            }
        }
        uint8_t* tile = btiles + (int64_t)(c0 / kChunk) * (cols * kChunk * 2);
        *reinterpret_cast<uint4*>(tile + tile_off(token, c0 % kChunk, kChunk)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(tile + tile_off(cols / 2 + token, c0 % kChunk, kChunk)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    };
#pragma unroll
    for (int i = 0; i < kPrepKeep; ++i) put((i * kPrepThreads + (int)threadIdx.x) * 8, keep[i]);
    for (int c0 = (kPrepKeep * kPrepThreads + (int)threadIdx.x) * 8; c0 < padded; c0 += kPrepThreads * 8) {
        float v[8];
        get(hr, c0, v);
        put(c0, v);
    }
}

__global__ void __launch_bounds__(kThreads, 1) lm_head_tc_kernel(const uint8_t* __restrict__ wtiles,
                                                                 const uint8_t* __restrict__ btiles, int64_t vocab,
                                                                 int hidden, int m, int cols, int stages, float* __restrict__ logits,
                                                                 unsigned int* err, bool w_f16, float cap) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int b_tile = cols * kChunk * 2, stage_bytes = kATile + b_tile;  // cols: hi | lo of the tokens, padded to 16 each
    uint8_t* stage_base = smem;  // stages x (A tile | B tile)
    uint64_t* full = reinterpret_cast<uint64_t*>(stage_base + (size_t)stages * stage_bytes);
    uint64_t* empty = full + kMaxStages;
    uint64_t* acc_full = empty + kMaxStages;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunks = (hidden + kChunk - 1) / kChunk;
    const int64_t row_sets = (vocab + kRows - 1) / kRows;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { ptx::mbar_init(&full[s], 1); ptx::mbar_init(&empty[s], 1); }
        ptx::mbar_init(acc_full, 1);
        ptx::mbar_init(acc_empty, 128);
        ptx::mbar_fence_init();
    }
    if (warp == 1) { ptx::tmem_alloc(tmem_slot, kCols); ptx::tmem_relinquish(); }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            // the weights of the first stages are requested before the wait on the kernel in front, which wrote the activations
            int ahead = 0;
            auto weights = [&](int64_t rs, int kc, int slot) {
                ptx::mbar_arrive_expect_tx(&full[slot], stage_bytes);
                ptx::bulk_g2s(stage_base + (size_t)slot * stage_bytes, wtiles + (rs * chunks + kc) * (int64_t)kATile, kATile, &full[slot]);
            };
            for (int64_t rs = blockIdx.x; rs < row_sets && ahead < stages; rs += gridDim.x)
                for (int kc = 0; kc < chunks && ahead < stages; ++kc, ++ahead) weights(rs, kc, ahead);
            ptx::pdl_wait();
            ptx::pdl_launch_dependents();
            int slot = 0, issued = 0; uint32_t par = 1; bool first = true;
            for (int64_t rs = blockIdx.x; rs < row_sets; rs += gridDim.x)
                for (int kc = 0; kc < chunks; ++kc) {
                    if (!first) ok &= ptx::mbar_wait_bounded(&empty[slot], par);
                    if (issued++ >= ahead) weights(rs, kc, slot);
                    ptx::bulk_g2s(stage_base + (size_t)slot * stage_bytes + kATile, btiles + (int64_t)kc * b_tile, b_tile, &full[slot]);
                    if (++slot == stages) { slot = 0; first = false; par ^= 1; }
                }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = instr_desc_bf16(kRows, cols, w_f16);
            int slot = 0; uint32_t par = 0, acc_par = 0; bool first_tile = true;
            for (int64_t rs = blockIdx.x; rs < row_sets; rs += gridDim.x) {
                if (!first_tile) { ok &= ptx::mbar_wait_bounded(acc_empty, acc_par); acc_par ^= 1; }
                first_tile = false;
                ptx::tc_fence_after();
                for (int kc = 0; kc < chunks; ++kc) {
                    ok &= ptx::mbar_wait_bounded(&full[slot], par);
                    ptx::tc_fence_after();
                    const uint32_t a_addr = ptx::smem_u32(stage_base + (size_t)slot * stage_bytes);
                    const uint32_t b_addr = a_addr + kATile;
#pragma unroll
                    for (int ks = 0; ks < kChunk / 16; ++ks) {  // K = 16 bf16 = 2 core matrices per MMA
                        const uint64_t ad = ptx::smem_desc(a_addr + ks * 256, 128, (kChunk / 8) * 128);
                        const uint64_t bd = ptx::smem_desc(b_addr + ks * 256, 128, (kChunk / 8) * 128);
                        ptx::umma_f16(tmem_base, ad, bd, idesc, (kc > 0 || ks > 0) ? 1u : 0u);
                    }
                    ptx::umma_commit(&empty[slot]);
                    if (++slot == stages) { slot = 0; par ^= 1; }
                }
                ptx::umma_commit(acc_full);
            }
        }
    } else {
        const int sub = warp & 3;
        uint32_t acc_par = 0;
        for (int64_t rs = blockIdx.x; rs < row_sets; rs += gridDim.x) {
            ok &= ptx::mbar_wait_bounded(acc_full, acc_par);
            acc_par ^= 1;
            ptx::tc_fence_after();
            const int64_t v = rs * kRows + sub * 32 + lane;
#pragma unroll 1
            for (int c0 = 0; c0 < cols / 2; c0 += 16) {
                uint32_t hi[16], lo[16];
                const uint32_t taddr = tmem_base + ((uint32_t)(sub * 32) << 16) + c0;
                ptx::tmem_ld16(taddr, hi);
                ptx::tmem_ld16(taddr + cols / 2, lo);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int token = c0 + j;
                    if (token < m && v < vocab) {
                        float r = __fadd_rn(__uint_as_float(hi[j]), __uint_as_float(lo[j]));
                        if (cap > 0.0f) r = cap * tanhf(r / cap);
                        logits[(int64_t)token * vocab + v] = r;
                    }
                }
            }
            ptx::tc_fence_before();
            ptx::mbar_arrive(acc_empty);
        }
    }
    if (!ok) atomicExch(err, kErrLmTimeout);
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) ptx::tmem_dealloc(tmem_base, kCols);
}

}  // namespace

size_t lm_head_tc_weight_bytes(int64_t vocab, int hidden) {
    return (size_t)((vocab + kRows - 1) / kRows) * ((hidden + kChunk - 1) / kChunk) * kATile;
}
size_t lm_head_tc_act_bytes(int hidden) { return (size_t)((hidden + kChunk - 1) / kChunk) * kBTile; }

cudaError_t launch_lm_retile(const __nv_bfloat16* w, int64_t vocab, int hidden, void* tiles, cudaStream_t stream, int ld) {
    lm_retile_kernel<<<1184, 256, 0, stream>>>(w, vocab, hidden, ld ? ld : hidden, reinterpret_cast<__nv_bfloat16*>(tiles));
    return cudaGetLastError();
}

// logits for up to 64 tokens per pass; h: [batch, hidden] residual stream (RMSNorm applied here)
cudaError_t launch_lm_head_tc(const void* wtiles, const float* h, const float* norm_w, float eps, int batch, int hidden,
                              int64_t vocab, void* btiles, float* logits, unsigned int* err, int sm_count,
                              cudaStream_t stream, bool w_f16, float cap) {
    constexpr size_t most = kRingBytes + 256;
    static PerDeviceOnce once;
    cudaError_t ce = once.run([] { return cudaFuncSetAttribute(lm_head_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most); });
    const int64_t row_sets = (vocab + kRows - 1) / kRows;
    const int grid = (int)(row_sets < sm_count ? row_sets : sm_count);
    for (int b0 = 0; b0 < batch && ce == cudaSuccess; b0 += kTok) {
        const int bc = batch - b0 < kTok ? batch - b0 : kTok;
        const int cols = (bc + 15) / 16 * 32, stage = kATile + cols * kChunk * 2;  // a product as wide as the tokens need
        const int stages = kRingBytes / stage < kMaxStages ? kRingBytes / stage : kMaxStages;
        ce = launch_pdl(lm_prep_kernel, dim3((unsigned)(cols / 2)), dim3(kPrepThreads), 0, stream, true, h + (size_t)b0 * hidden, norm_w, eps, hidden, bc, cols,
                        reinterpret_cast<uint8_t*>(btiles), w_f16);
        if (ce == cudaSuccess)
            ce = launch_pdl(lm_head_tc_kernel, dim3((unsigned)grid), dim3(kThreads), (size_t)stages * stage + 256, stream, true, reinterpret_cast<const uint8_t*>(wtiles),
                            reinterpret_cast<const uint8_t*>(btiles), vocab, hidden, bc, cols, stages, logits + (size_t)b0 * vocab, err, w_f16, cap);
    }
    return ce;
}

}  // namespace bt

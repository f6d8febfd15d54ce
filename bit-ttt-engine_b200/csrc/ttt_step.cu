// One decode step of a small TTT model, embedding to residual stream, in one launch: one cluster of eight CTAs, which hold the
// stream and the vectors between the layers' stages in shared memory, every CTA all of them.
// A stage (down, fast-weight update, up, gate|up, down) is a product of a few row tiles or the update of a few rows: as launches of
// their own the 5 stages of a layer took 4 us each, start-up, wait for the kernel in front and trips to L2, whatever the
// arithmetic.  Here a CTA takes every eighth row tile, stores its results into all eight CTAs' shared memory, and a cluster
// barrier ends the stage; weights and norm weights of the next stage are requested in front of the barrier.
// Bound by that chain of stages, 2.5 us each (barrier, activations quantised by every CTA, one or two tiles a warp): 256 x 64, ff 688,
// four layers, one sequence: 50 us a step, of which the launches took 84.
// Same arithmetic as the launches it stands for (gemv.cu, ttt.cu, glue.cu): integer products, f32 elsewhere in the same order,
// f64 sums of squares rounded once.
#include "bt_model.cuh"
#include "bt_ptx.cuh"
#include "bt_tile_mma.cuh"

namespace bt {

namespace {

constexpr int kCtas = 8, kStepThreads = 512, kStepWarps = kStepThreads / 32;
constexpr int kMaxTokens = 8, kMaxHidden = 512, kMaxSmall = 128, kMaxFf = 2048;
constexpr int kTilesPerWarp = 4;   // gate|up of the largest sizes: 256 row tiles x 2, over 8 CTAs of 16 warps
constexpr int kGroups = 8;         // groups of four values a thread quantises at most: 2048 values, 64 threads a token
constexpr int kRowTiles = kMaxFf * 2 / kTileRows / kCtas;

struct __align__(16) StepSmem {
    float h[kMaxTokens][kMaxHidden];     // residual stream
    float feat[kMaxTokens][kMaxSmall];   // down-projected features, then predictions
    float z[kMaxTokens][kMaxSmall];
    float act[kMaxTokens][kMaxFf];       // silu(gate) * up
    uint8_t image[kMaxTokens][kMaxFf + 64];  // int8 activations as the B operand wants them
    float xs[kMaxTokens][kMaxSmall + 4 * (kMaxSmall / 16)];  // normalised features
    int acc[kRowTiles][128];             // sums of the row tiles: [4 accumulator registers][32 lanes]
    double red_d[kStepWarps];
    float red_f[kStepWarps];
    float sx[kMaxTokens];
    int qsum[kMaxTokens];
};

__device__ __forceinline__ float get16(const __nv_bfloat16* p, bool f16) {
    return f16 ? __half2float(*reinterpret_cast<const __half*>(p)) : __bfloat162float(*p);
}

template <int D>  // width of the fast weights: 32, 64 or 128
__global__ void __launch_bounds__(kStepThreads, 1) ttt_step_kernel(const TttStepArgs a) {
    constexpr int LPR = D / 16, kRowsPerPass = 32 / LPR, kPad = 4, H = 4 * D;
    extern __shared__ __align__(16) uint8_t raw[];
    StepSmem& sm = *reinterpret_cast<StepSmem*>(raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = (int)ptx::cluster_ctarank();
    const int B = a.batch, I = a.ff;
    const int slots = B <= 1 ? 1 : (B <= 2 ? 2 : (B <= 4 ? 4 : 8)), per = kStepThreads / slots;  // threads of a token in the quantisers
    const int my_token = tid / per, sub = tid - my_token * per;
    uint32_t window[kCtas];
#pragma unroll
    for (int r = 0; r < kCtas; ++r) window[r] = ptx::map_to_rank(raw, (uint32_t)r);
    auto push = [&](float* at, float v) {  // into every CTA's shared memory
        const uint32_t off = ptx::smem_u32(at) - ptx::smem_u32(raw);
#pragma unroll
        for (int r = 0; r < kCtas; ++r) ptx::st_dsmem_f32(window[r] + off, v);
    };

    // ---- weights of a stage, requested ahead ----
    uint4 w4[kTilesPerWarp], v4[kTilesPerWarp];
    float2 sw;  // weight scales of rows 0-7 and 8-15 of a row tile: the same in every tile of these matrices (gate and up differ)
    auto request = [&](const uint8_t* tiles, const float* scales, int row_tiles, int k_tiles) {
        sw = make_float2(__ldg(scales), __ldg(scales + 1));
        const int total = (row_tiles - cta + kCtas - 1) / kCtas * k_tiles;
#pragma unroll
        for (int u = 0; u < kTilesPerWarp; ++u) {
            const int i = warp + u * kStepWarps;
            if (i < total) {
                const int lt = i / k_tiles, kt = i - lt * k_tiles;
                const uint8_t* p = tiles + ((int64_t)(cta + lt * kCtas) * k_tiles + kt) * kTileBytes + lane * 16;
                w4[u] = __ldg(reinterpret_cast<const uint4*>(p));
                v4[u] = __ldg(reinterpret_cast<const uint4*>(p + 512));
            }
        }
    };
    float4 nw[2];
    auto request_norm = [&](const float* w) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int g = sub + i * per;
            if (g < H / 4) nw[i] = __ldg(reinterpret_cast<const float4*>(w + 4 * g));
        }
    };
    // ---- rows of `src` (stride ld, k values) to int8; norm: RMSNorm with the weights in nw first ----
    auto quantise = [&](const float* src, int ld, int k, bool norm) {
        const int groups = k >> 2, groups_pad = (k + kTileK - 1) / kTileK * (kTileK / 4);
        const int token_warp0 = my_token * (per / 32), token_warps = per / 32;
        const bool live = my_token < B;
        if (tid < kMaxTokens) sm.qsum[tid] = 0;
        float4 v[kGroups];
#pragma unroll
        for (int i = 0; i < kGroups; ++i) {
            const int g = sub + i * per;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && g < groups) v[i] = *reinterpret_cast<const float4*>(src + my_token * ld + 4 * g);
        }
        if (norm) {
            double ss = 0.0;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                ss = fma((double)v[i].x, (double)v[i].x, ss); ss = fma((double)v[i].y, (double)v[i].y, ss);
                ss = fma((double)v[i].z, (double)v[i].z, ss); ss = fma((double)v[i].w, (double)v[i].w, ss);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) sm.red_d[warp] = ss;
            __syncthreads();
            ss = (lane & 15) < token_warps ? sm.red_d[token_warp0 + (lane & 15)] : 0.0;  // (a loop over them took 16 trips to shared memory)
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float denom = sqrtf(__fadd_rn((float)(ss / (double)k), a.eps));
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (sub + i * per < groups) {
                    v[i].x = __fmul_rn(__fdiv_rn(v[i].x, denom), nw[i].x); v[i].y = __fmul_rn(__fdiv_rn(v[i].y, denom), nw[i].y);
                    v[i].z = __fmul_rn(__fdiv_rn(v[i].z, denom), nw[i].z); v[i].w = __fmul_rn(__fdiv_rn(v[i].w, denom), nw[i].w);
                }
        }
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < kGroups; ++i) amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v[i].x), fabsf(v[i].y))), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (lane == 0) sm.red_f[warp] = amax;
        __syncthreads();
        amax = (lane & 15) < token_warps ? sm.red_f[token_warp0 + (lane & 15)] : 0.0f;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
        int local = 0;
#pragma unroll
        for (int i = 0; i < kGroups; ++i) {
            if (i * per >= groups_pad) break;
            const int g = sub + i * per;  // values 4 g .. 4 g + 3: byte g % 4 of the words of 16-group g / 4
            if (live && g < groups_pad) {
                int q[4] = {ptx::round_half_away(__fmul_rn(v[i].x, inv)), ptx::round_half_away(__fmul_rn(v[i].y, inv)),
                            ptx::round_half_away(__fmul_rn(v[i].z, inv)), ptx::round_half_away(__fmul_rn(v[i].w, inv))};
                const uint32_t word = ptx::pack4_sat_s8(q[0], q[1], q[2], q[3]);
                local = ptx::dp4a_s8s8(word, 0x01010101u, local);
                const int j = g >> 2;
                uint8_t* p = sm.image[my_token] + (j >> 4) * kTileK + ((j >> 2) & 3) * 16 + (j & 3) * 4 + (g & 3);
#pragma unroll
                for (int r = 0; r < 4; ++r) p[r * 64] = (uint8_t)(word >> (8 * r));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
        if (lane == 0 && live) atomicAdd(&sm.qsum[my_token], local);
        if (sub == 0 && live) sm.sx[my_token] = __fdiv_rn(amax, 127.0f);
        __syncthreads();
    };
    // ---- this CTA's row tiles times the image; the sums of row tile lt (of this CTA) in sm.acc[lt] ----
    auto multiply = [&](int row_tiles, int k_tiles) {
        const int total = (row_tiles - cta + kCtas - 1) / kCtas * k_tiles;
        const int g = lane >> 2, t = lane & 3;
        const uint8_t* acts = sm.image[g < B ? g : B - 1] + t * 16;
#pragma unroll
        for (int u = 0; u < kTilesPerWarp; ++u) {
            const int i = warp + u * kStepWarps;
            if (i < total) {
                const int lt = i / k_tiles, kt = i - lt * k_tiles;
                uint4 b4[4];
                int acc[4][4];
#pragma unroll
                for (int f = 0; f < 4; ++f) b4[f] = lds128(acts + kt * kTileK + f * 64);
                tile_mma_r<true>(acc, w4[u], v4[u], b4);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    red_add_s32(&sm.acc[lt][j * 32 + lane], acc[0][j] + (acc[1][j] >> 2) + (acc[2][j] >> 4) + (acc[3][j] >> 6));
            }
        }
        __syncthreads();
    };
    auto sum_of = [&](int lt, int row, int token) -> int {
        return sm.acc[lt][((row >> 3) * 2 + (token & 1)) * 32 + (row & 7) * 4 + (token >> 1)] - sm.qsum[token];
    };
    // f(row of the matrix, token, (sum - sum q) * s_w * s_x) for this CTA's rows below n
    auto each_output = [&](int row_tiles, int n, auto f) {
        const int rts = (row_tiles - cta + kCtas - 1) / kCtas;
        for (int i = tid; i < rts * kTileRows * B; i += kStepThreads) {
            const int token = i / (rts * kTileRows), e = i - token * (rts * kTileRows), lt = e / kTileRows, r = e % kTileRows;
            const int row = (cta + lt * kCtas) * kTileRows + r;
            if (row < n) f(row, token, __fmul_rn(__fmul_rn((float)sum_of(lt, r, token), r < 8 ? sw.x : sw.y), sm.sx[token]));
        }
    };

    const int h_tiles = (H + kTileK - 1) / kTileK, i_tiles = (I + kTileK - 1) / kTileK;
    const int rt_small = (D + kTileRows - 1) / kTileRows, rt_h = H / kTileRows, rt_gu = (2 * I + kTileRows - 1) / kTileRows;
    auto clear = [&]() {  // the sums of every row tile (columns without a token hold the last token's)
        for (int i = tid; i < (max(rt_gu, rt_h) - cta + kCtas - 1) / kCtas * 128; i += kStepThreads) (&sm.acc[0][0])[i] = 0;
    };
    clear();
    const TttStepLayer* L = a.layers;
    request(L->down, L->sw_down, rt_small, h_tiles);
    request_norm(L->norm1);
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    for (int i = tid; i < B * H; i += kStepThreads) {
        const int b = i / H, c = i - b * H;
        int tok = a.tokens[b];
        tok = tok < 0 ? 0 : (tok >= a.vocab ? a.vocab - 1 : tok);
        sm.h[b][c] = get16(a.embed + (int64_t)tok * H + c, a.f16);
    }
    ptx::cluster_arrive();  // every CTA of the cluster runs: its shared memory may be written
    ptx::cluster_wait();

    // fast weights: warp pass p (rows p * kRowsPerPass .. of the batch's states) belongs to CTA p % 8, warp p / 8 % 16
    const int passes = B * D / kRowsPerPass, blk = lane % LPR;
    auto state_row = [&](float* w, int p) { return w + ((int64_t)p * kRowsPerPass + lane / LPR) * D + blk * 16; };
    auto barrier = [&]() { ptx::cluster_arrive(); ptx::cluster_wait(); };

    for (int li = 0; li < a.num_layers; ++li, ++L) {
        // ---- features = down(norm1(h)) ----
        quantise(&sm.h[0][0], kMaxHidden, H, true);
        multiply(rt_small, h_tiles);
        each_output(rt_small, D, [&](int row, int token, float y) { push(&sm.feat[token][row], y); });
        const int p0 = cta + warp * kCtas;
        float4 wr[4];
        if (p0 < passes) {
#pragma unroll
            for (int i = 0; i < 4; ++i) wr[i] = reinterpret_cast<const float4*>(state_row(L->w_state, p0))[i];
        }
        request(L->up, L->sw_up, rt_h, 1);
        __syncthreads();
        clear();
        barrier();
        // ---- fast weights: x = f / (|f| + 1e-6), z = W x, W <- W - lr (z - x) x^T (layers/ttt.rs:48-74) ----
        {
            const int t = tid >> 4, s16 = tid & 15;  // 16 threads a token
            if (t < kMaxTokens) {                    // (whole warps)
                float f[LPR];
                double ss = 0.0;
#pragma unroll
                for (int e = 0; e < LPR; ++e) f[e] = t < B ? sm.feat[t][s16 + 16 * e] : 0.0f;
#pragma unroll
                for (int e = 0; e < LPR; ++e) ss = fma((double)f[e], (double)f[e], ss);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                const float nrm = __fadd_rn(sqrtf((float)ss), 1e-6f);
#pragma unroll
                for (int e = 0; e < LPR; ++e)
                    if (t < B) sm.xs[t][s16 + (16 + kPad) * e] = __fdiv_rn(f[e], nrm);
            }
            __syncthreads();
            for (int p = p0; p < passes; p += kCtas * kStepWarps) {
                float* wp = state_row(L->w_state, p);
                if (p != p0) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) wr[i] = reinterpret_cast<const float4*>(wp)[i];
                }
                const int row_all = p * kRowsPerPass + lane / LPR, b = row_all / D, row = row_all - b * D;
                const float* xt = sm.xs[b];
                float x[16], w[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 v = *reinterpret_cast<const float4*>(xt + blk * (16 + kPad) + 4 * i);
                    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
                    w[4 * i] = wr[i].x; w[4 * i + 1] = wr[i].y; w[4 * i + 2] = wr[i].z; w[4 * i + 3] = wr[i].w;
                }
                float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    s0 = __fmaf_rn(w[i], x[i], s0); s1 = __fmaf_rn(w[i + 1], x[i + 1], s1);
                    s2 = __fmaf_rn(w[i + 2], x[i + 2], s2); s3 = __fmaf_rn(w[i + 3], x[i + 3], s3);
                }
                float s = __fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3));
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
                const float df = __fsub_rn(s, xt[row + kPad * (row / 16)]);
                if (blk == 0) push(&sm.z[b][row], s);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float4 v;
                    v.x = __fsub_rn(w[4 * i], __fmul_rn(__fmaf_rn(df, x[4 * i], 0.0f), a.lr));
                    v.y = __fsub_rn(w[4 * i + 1], __fmul_rn(__fmaf_rn(df, x[4 * i + 1], 0.0f), a.lr));
                    v.z = __fsub_rn(w[4 * i + 2], __fmul_rn(__fmaf_rn(df, x[4 * i + 2], 0.0f), a.lr));
                    v.w = __fsub_rn(w[4 * i + 3], __fmul_rn(__fmaf_rn(df, x[4 * i + 3], 0.0f), a.lr));
                    reinterpret_cast<float4*>(wp)[i] = v;
                }
            }
        }
        barrier();
        // ---- h += up(z) ----
        quantise(&sm.z[0][0], kMaxSmall, D, false);
        multiply(rt_h, 1);
        each_output(rt_h, H, [&](int row, int token, float y) { push(&sm.h[token][row], __fadd_rn(sm.h[token][row], y)); });
        request(L->gate_up, L->sw_gate_up, rt_gu, h_tiles);
        request_norm(L->norm2);
        __syncthreads();
        clear();
        barrier();
        // ---- act = silu(gate(norm2(h))) * up(norm2(h)): rows 0-7 of a tile are gate rows, rows 8-15 the matching up rows ----
        quantise(&sm.h[0][0], kMaxHidden, H, true);
        multiply(rt_gu, h_tiles);
        {
            const int rts = (rt_gu - cta + kCtas - 1) / kCtas;
            for (int i = tid; i < rts * 8 * B; i += kStepThreads) {
                const int token = i / (rts * 8), e = i - token * (rts * 8), lt = e >> 3, r = e & 7, col = (cta + lt * kCtas) * 8 + r;
                if (col < I) {
                    const float y = __fmul_rn(__fmul_rn((float)sum_of(lt, r, token), sw.x), sm.sx[token]);
                    const float uv = __fmul_rn(__fmul_rn((float)sum_of(lt, r + 8, token), sw.y), sm.sx[token]);
                    push(&sm.act[token][col], __fmul_rn(__fdiv_rn(y, __fadd_rn(1.0f, expf(-y))), uv));  // layers/swiglu.rs:31-33
                }
            }
        }
        request(L->mlp_down, L->sw_mlp_down, rt_h, i_tiles);
        __syncthreads();
        clear();
        barrier();
        // ---- h += down(act) ----
        quantise(&sm.act[0][0], kMaxFf, I, false);
        multiply(rt_h, i_tiles);
        each_output(rt_h, H, [&](int row, int token, float y) { push(&sm.h[token][row], __fadd_rn(sm.h[token][row], y)); });
        if (li + 1 < a.num_layers) {
            request(L[1].down, L[1].sw_down, rt_small, h_tiles);
            request_norm(L[1].norm1);
        }
        __syncthreads();
        clear();
        barrier();
    }
    for (int i = cta * kStepThreads + tid; i < B * H; i += kCtas * kStepThreads) a.h[i] = sm.h[i / H][i % H];
}

}  // namespace

// Up to eight sequences (the columns of an MMA) of a model whose vectors all fit a CTA's shared memory; sizes whose fast weights the
// row form of the update takes (d = 32, 64, 128).  Wider models have work for more than the eight SMs of a cluster in each stage.
bool ttt_step_fits(int hidden, int small, int ff, int batch) {
    return (small == 32 || small == 64 || small == 128) && hidden == 4 * small && ff <= kMaxFf && ff % 16 == 0 && batch >= 1 && batch <= kMaxTokens;
}

cudaError_t launch_ttt_model_step(const TttStepArgs& a, int small, cudaStream_t s) {
    if (!ttt_step_fits(a.hidden, small, a.ff, a.batch)) return cudaErrorInvalidValue;
    auto* kernel = small == 32 ? ttt_step_kernel<32> : (small == 64 ? ttt_step_kernel<64> : ttt_step_kernel<128>);
    static PerDeviceOnce once;
    cudaError_t e = once.run([] {
        cudaError_t r = cudaFuncSetAttribute(ttt_step_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StepSmem));
        if (r == cudaSuccess) r = cudaFuncSetAttribute(ttt_step_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StepSmem));
        if (r == cudaSuccess) r = cudaFuncSetAttribute(ttt_step_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StepSmem));
        return r;
    });
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCtas);
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = sizeof(StepSmem);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCtas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

}  // namespace bt

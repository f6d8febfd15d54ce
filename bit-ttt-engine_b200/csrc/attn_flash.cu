// Prompt attention over a bf16 cache on tcgen05: a CTA owns 128 query positions of one head and walks tiles of 128 keys.
//   S = Q K^T (both K-major in shared memory, f32 in tensor memory), P = exp2(score(S) - reference) as bf16 hi + lo over the
//   scores' own columns, O += P V (P the A operand in tensor memory, V MN-major as its rows lie).
// Warps: 8 softmax (two groups of four: group w takes the key tiles w, w + 2, ..., a thread one query row = one tensor-memory
// lane), 4 loaders, 1 MMA.  Each group has scores, maxima, sums and output accumulators of its own, so that the MMAs of one
// tile run under the other group's softmax; the two halves meet at the end.
// A row's reference is the largest score so far, moved only when it grows by more than 2^8: the accumulators in tensor memory
// are rescaled a few times per prompt instead of once per tile, and weights stay below 2^8 (their hi + lo keep 16 significand
// bits whatever the power of two).
// Bound: the special-function unit (ex2 per score, with a score cap ex2 + rcp + ex2: 3 x 16384 of 16 a clock and tile = 3072
// clocks, against 770 of MMAs for heads of 64), then the softmax warps' instructions.
// 1999 tokens, us a layer, with mma.sync tiles of 64 x 64 before -> now: 32 heads of 64 with a cap 175 -> 92, 16 heads of 192 + 128
// 279 -> 59.  What is left beside the loop is a CTA's beginning and end and the last round of CTAs.  Every second exponential by a
// polynomial on the FMA units: 130 -> 155 at the time (the softmax warps are bound by issue too).  Warpgroups that trade registers
// (no spills of the 128 of a launch): 117 -> 112.
#include <type_traits>

#include "attn_dense.cuh"
#include "bt_ptx.cuh"

namespace bt {

namespace {

constexpr int kFlashQ = 128, kFlashKeys = 128, kSoftmaxWarps = 8, kFlashLoaders = 4;
constexpr int kMmaWarp = kSoftmaxWarps + kFlashLoaders;
constexpr int kFlashThreads = (kMmaWarp + 4) * 32;  // whole warpgroups, which trade registers: three warps behind the MMA warp idle
constexpr int kRegsSoftmax = 184, kRegsLoad = 80, kRegsMma = 56;
constexpr int kRegsShares = 256 * kRegsSoftmax + 128 * kRegsLoad + 128 * kRegsMma;
static_assert(kRegsShares <= kFlashThreads * 128, "a launch of 512 threads has 128 registers each at most");
constexpr int kFlashMaxK = 192, kFlashMaxV = 128;
constexpr unsigned kErrFlashTimeout = 0x46415454u;  // 'FATT'
constexpr float kGrow = 8.0f;                       // how far (log2) a score may exceed its row's reference
constexpr float kNone = -INFINITY;

// f32 += bf16 . bf16, M = 128; b_mn: B is MN-major
__device__ __forceinline__ uint32_t flash_idesc(int n, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}

// the loads into v are complete (v is named, so that no use of it is moved before the wait)
__device__ __forceinline__ void ld_wait32(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                   "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]),
                   "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]),
                   "+r"(v[30]), "+r"(v[31])
                 :: "memory");
}
// f(c0, v) on 32 columns after 32 of a lane's 128.  Rolled up, and without the next columns on their way: unrolled four times, with the
// loads ahead, the softmax did not stay in the instruction caches (no_instruction 2 of 6.5 stalled warps an issue): 111 us a layer of
// 32 heads of 64 with a cap, 99 unrolled twice, 92 like this, and no better with the loads ahead in a rolled loop (95).
template <typename F>
__device__ __forceinline__ void each_32(uint32_t addr, F f) {
#pragma unroll 1
    for (int c0 = 0; c0 < kFlashKeys; c0 += 32) {
        uint32_t v[32];
        ptx::tmem_ld32(addr + c0, v);
        ld_wait32(v);
        f(c0, v);
    }
}

struct FlashSmem {  // behind the operands
    uint64_t k_full[2], v_full[2], s_full[3], p_full[2], o_done[2];
    float m[2][kFlashQ], l[2][kFlashQ];
    uint32_t tmem;
};
// Operands: [16-byte piece of a row][row] 16 bytes, a core matrix (8 rows) is 128 contiguous bytes
__host__ __device__ constexpr size_t flash_bytes(int k_steps, int v_steps) {
    return (size_t)(3 * k_steps + 2 * v_steps) * 2 * kFlashKeys * 16;
}
constexpr int kFlashSmemMost = 227 * 1024;
static_assert(flash_bytes(kFlashMaxK / 16, kFlashMaxV / 16) + sizeof(FlashSmem) <= kFlashSmemMost, "the largest heads fit shared memory");

template <bool LATENT, bool CAP>
__global__ void __launch_bounds__(kFlashThreads, 1) attn_flash_kernel(const DenseAttn a, const LatentTile lt, const ActOut out) {
    extern __shared__ __align__(128) uint8_t fsm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ks = a.kv.k_stride, vs = a.kv.v_stride;
    const int nk = (ks + 15) / 16, nv = (vs + 15) / 16;                 // 16-wide steps
    const uint32_t k_bytes = (uint32_t)nk * 2 * kFlashKeys * 16, v_bytes = (uint32_t)nv * 2 * kFlashKeys * 16;
    uint8_t* q_s = fsm;
    uint8_t* k_s = q_s + k_bytes;                                       // two tiles
    uint8_t* v_s = k_s + 2 * k_bytes;
    FlashSmem& sm = *reinterpret_cast<FlashSmem*>(v_s + 2 * v_bytes);

    const int qt = gridDim.y - 1 - blockIdx.y;                          // the longest first, of every head
    const int head = blockIdx.x, b = blockIdx.z + (LATENT ? lt.b0 : 0), g = LATENT ? 0 : head / (a.heads / a.n_kv);
    const int past = a.pos[b], q0 = qt * kFlashQ, rows = min(kFlashQ, a.q_rows - q0);
    const int last = past + q0 + rows - 1;                              // last position any row of this tile sees
    const int tiles = last / kFlashKeys + 1;

    if (warp == 0 && lane < 2) {
        ptx::mbar_init(&sm.k_full[lane], kFlashLoaders / 2 * 32);
        ptx::mbar_init(&sm.v_full[lane], kFlashLoaders / 2 * 32);
        ptx::mbar_init(&sm.s_full[lane], 1);
        if (lane == 0) ptx::mbar_init(&sm.s_full[2], 1);
        ptx::mbar_init(&sm.p_full[lane], 4);
        ptx::mbar_init(&sm.o_done[lane], 1);
        ptx::mbar_fence_init();
    }
    if (warp == kMmaWarp) { ptx::tmem_alloc(&sm.tmem, 512); ptx::tmem_relinquish(); }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    // Tensor memory: places of 128 columns for a tile's scores (its weights afterwards), tile t's t mod places, then the groups'
    // outputs.  Values of up to 64 columns leave room for a third place: the scores of tile t + 2 are then made during the softmax
    // of tile t, while with two they wait for the product that reads tile t's weights (2 000 clocks of a group's 9 200).
    const int places = nv <= kFlashMaxV / 32 ? 3 : 2, o_cols = places == 3 ? kFlashMaxV / 2 : kFlashMaxV;
    const uint32_t tmem = sm.tmem, tmem_o = tmem + places * kFlashKeys;
    auto place_of = [&](int t) { return places == 3 ? t % 3 : t & 1; };
    auto scores_made = [&](int t) -> bool { return ptx::mbar_wait_bounded(&sm.s_full[place_of(t)], (uint32_t)((places == 3 ? t / 3 : t >> 1) & 1)); };
    bool ok = true;

    if (warp >= kSoftmaxWarps && warp < kMmaWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsLoad));
        // ---------------- loaders: two warps bring keys (the queries with the first tile), two bring values ----------------
        // Apart, because a tile's keys are wanted as soon as their place is free, which is half a tile's softmax before the
        // values' place is: in one sequence the next scores waited for the copies of values behind them.
        const int lw = (warp - kSoftmaxWarps) & 1, r8 = lane & 7, c4 = lane >> 3;
        const bool keys = warp - kSoftmaxWarps < 2;
        constexpr int kPiece = kFlashKeys * 16;
        const uint8_t* q_src = reinterpret_cast<const uint8_t*>(a.q_buf) + ((((int64_t)b * a.q_rows + q0) * a.heads + head) * ks) * 2;
        // A warp instruction copies 8 rows x 4 pieces: whole core matrices in shared memory, 64 bytes of a row in global memory.
        // Pieces p0 .. p1 of 128 rows, of which `rows` exist (the others, and pieces from `live` on, become zeros); row r and piece p
        // lie at src + r / 8 * group + r % 8 * row + (p - p0) * piece.  One address a row group: computed for every copy they took
        // 125 to 212 clocks each (fepapel's keys 10 300 a tile).
        auto copy = [&](uint8_t* dst, int p0, int p1, int live, int rows, const uint8_t* src, int64_t group, int64_t row, int piece) {
            uint32_t to = ptx::smem_u32(dst) + (p0 + c4) * kPiece + (lw * 8 + r8) * 16;
            const uint8_t* from = src + lw * group + r8 * row + c4 * piece;
            if (rows >= kFlashKeys && live >= p1) {  // every tile but the last: nothing to ask about a copy
                for (int p = p0 + c4; p < p1; p += 4, to += 4 * kPiece, from += 4 * piece) {
                    const uint8_t* f = from;
#pragma unroll
                    for (int i = 0; i < kFlashKeys / 16; ++i, f += 2 * group) ptx::cp16(to + i * 256, f, true);
                }
                return;
            }
            for (int r = lw * 8 + r8; r < kFlashKeys; r += 16, to += 16 * 16, from += 2 * group) {
                const bool there = r < rows;
#pragma unroll 4
                for (int p = 0; p < p1 - p0 - c4; p += 4) {
                    const bool on = there && p0 + c4 + p < live;
                    ptx::cp16(to + p * kPiece, on ? from + p * piece : q_src, on);
                }
            }
        };
        const int k_main = LATENT ? lt.k_main : ks;  // columns of a head's own keys
        const uint8_t* k_src = LATENT ? reinterpret_cast<const uint8_t*>(lt.kv + blockIdx.z * lt.kv_seq + head * lt.k_main)
                                      : reinterpret_cast<const uint8_t*>(a.kv.k) + ((int64_t)b * a.n_kv + g) * a.kv.max_seq * ks * 2;
        const uint8_t* v_src = LATENT ? reinterpret_cast<const uint8_t*>(lt.kv + blockIdx.z * lt.kv_seq + a.heads * lt.k_main + head * vs)
                                      : reinterpret_cast<const uint8_t*>(a.kv.v) + ((int64_t)b * a.n_kv + g) * a.kv.max_seq * vs * 2;
        const int64_t k_row = 2 * (LATENT ? lt.kv_ld : ks), v_row = 2 * (LATENT ? lt.kv_ld : vs), rot_group = (int64_t)lt.latent.cols() * 16;
        const uint8_t* rot_src = LATENT ? reinterpret_cast<const uint8_t*>(lt.latent.rows) + b * lt.latent.seq_bytes() + lt.latent.off(0, lt.latent.rot_col()) : nullptr;
        auto load_k = [&](int t) {
            uint8_t* dst = k_s + (t & 1) * k_bytes;
            const int rows = last + 1 - t * kFlashKeys;
            copy(dst, 0, LATENT ? k_main / 8 : 2 * nk, k_main / 8, rows, k_src + (int64_t)t * kFlashKeys * k_row, 8 * k_row, k_row, 16);
            if (LATENT) copy(dst, k_main / 8, 2 * nk, ks / 8, rows, rot_src + (int64_t)t * (kFlashKeys / 8) * rot_group, rot_group, 16, 128);
        };
        auto load_v = [&](int t) {
            copy(v_s + (t & 1) * v_bytes, 0, 2 * nv, vs / 8, last + 1 - t * kFlashKeys, v_src + (int64_t)t * kFlashKeys * v_row, 8 * v_row, v_row, 16);
        };
        auto publish = [&](uint64_t* bar) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            ptx::fence_async_smem();
            ptx::mbar_arrive(bar);
        };
        if (keys) copy(q_s, 0, 2 * nk, ks / 8, rows, q_src, (int64_t)8 * a.heads * ks * 2, (int64_t)a.heads * ks * 2, 16);
        for (int t = 0; t < tiles; ++t) {
            // the tile's place: the scores of tile t - 2 are made, or its values are multiplied
            if (t >= 2) ok &= keys ? scores_made(t - 2) : ptx::mbar_wait_bounded(&sm.o_done[t & 1], (uint32_t)(((t - 2) >> 1) & 1));
            if (keys) load_k(t);
            else load_v(t);
            publish(keys ? &sm.k_full[t & 1] : &sm.v_full[t & 1]);
        }
    } else if (warp >= kMmaWarp) {
        // ---------------- MMA ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsMma));
        if (warp == kMmaWarp && lane == 0) {
            const uint32_t qk = flash_idesc(kFlashKeys, false), pv = flash_idesc(16 * nv, true);
            constexpr uint32_t kPiece = kFlashKeys * 16;
            const uint64_t qd = ptx::smem_desc(ptx::smem_u32(q_s), kPiece, 128);
            const uint64_t kd0 = ptx::smem_desc(ptx::smem_u32(k_s), kPiece, 128), vd0 = ptx::smem_desc(ptx::smem_u32(v_s), 128, kPiece);
            auto scores = [&](int t) {
                const int w = t & 1;
                ok &= ptx::mbar_wait_bounded(&sm.k_full[w], (uint32_t)((t >> 1) & 1));
                ptx::tc_fence_after();
                const uint64_t kd = kd0 + w * (k_bytes >> 4);
                for (int k = 0; k < nk; ++k)  // (a descriptor counts in units of 16 bytes)
                    ptx::umma_f16(tmem + place_of(t) * kFlashKeys, qd + k * (2 * kPiece >> 4), kd + k * (2 * kPiece >> 4), qk, k > 0 ? 1u : 0u);
                ptx::umma_commit(&sm.s_full[place_of(t)]);
            };
            for (int t = 0; t < places && t < tiles; ++t) scores(t);
            for (int t = 0; t < tiles; ++t) {
                const int w = t & 1;
                ok &= ptx::mbar_wait_bounded(&sm.v_full[w], (uint32_t)((t >> 1) & 1));
                ok &= ptx::mbar_wait_bounded(&sm.p_full[w], (uint32_t)((t >> 1) & 1));
                ptx::tc_fence_after();
                const uint64_t vd = vd0 + w * (v_bytes >> 4);
                const uint32_t p = tmem + place_of(t) * kFlashKeys, o = tmem_o + w * o_cols;
                // 32 keys' weights lie over their scores: 16 columns hi, 16 columns lo; 16 keys are 256 bytes of V further on
#pragma unroll
                for (int k = 0; k < kFlashKeys / 16; ++k) {
                    const uint32_t pk = p + (k >> 1) * 32 + (k & 1) * 8;
                    ptx::umma_f16_ts(o, pk, vd + k * 16, pv, t >= 2 || k > 0 ? 1u : 0u);
                    ptx::umma_f16_ts(o, pk + 16, vd + k * 16, pv, 1u);
                }
                ptx::umma_commit(&sm.o_done[w]);
                if (t + places < tiles) scores(t + places);  // (MMAs run in order: these write the columns that the ones above read)
            }
        }
    } else {
        // ---------------- softmax ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
        const int w = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const uint32_t o_tm = tmem_o + lanes;
        const ScoreMap score(a.scale, a.softcap);
        const float half_cap = 0.5f * score.cap2;
        float m_ref = kNone, l0 = 0.0f, l1 = 0.0f;
        for (int t = w; t < tiles; t += 2) {
            ok &= scores_made(t);
            ptx::tc_fence_after();
            const uint32_t s_tm = tmem + lanes + place_of(t) * kFlashKeys;
            const int seen = past + q0 + r - t * kFlashKeys;                                        // keys 0 .. seen of the tile are visible
            const bool mask = past + q0 + quarter * 32 < t * kFlashKeys + kFlashKeys - 1;            // (one answer per warp)
            // largest raw score (the map is monotonic, scale > 0)
            float mx0 = kNone, mx1 = kNone;
            each_32(s_tm, [&](int c0, uint32_t (&v)[32]) {
                if (mask) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = c0 + j <= seen ? v[j] : __float_as_uint(kNone);
                }
#pragma unroll
                for (int j = 0; j < 32; j += 2) { mx0 = fmaxf(mx0, __uint_as_float(v[j])); mx1 = fmaxf(mx1, __uint_as_float(v[j + 1])); }
            });
            const float raw = fmaxf(mx0, mx1);
            const float top = raw == kNone ? kNone : score(raw);
            if (t < 2) {
                m_ref = top;
            } else {
                const bool grows = top > m_ref + kGrow;
                if (__any_sync(0xffffffffu, grows)) {
                    const float al = grows ? ex2(m_ref - top) : 1.0f;  // (nothing seen so far: 0)
                    ok &= ptx::mbar_wait_bounded(&sm.o_done[w], (uint32_t)(((t - 2) >> 1) & 1));
                    ptx::tc_fence_after();
                    for (int c0 = 0; c0 < 16 * nv; c0 += 16) {
                        uint32_t v[16];
                        ptx::tmem_ld16(o_tm + w * o_cols + c0, v);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * al);
                        ptx::tmem_st16(o_tm + w * o_cols + c0, v);
                    }
                    l0 *= al;
                    l1 *= al;
                    if (grows) m_ref = top;
                }
            }
            const float ref = m_ref == kNone ? 0.0f : m_ref;  // (no key visible yet: every weight is 0)
            const float shift = CAP ? half_cap - ref : -ref;
            // (one copy of the loop for tiles that the diagonal crosses and one for the others: a mask costs every score two instructions)
            auto weights = [&](auto masked) {
            each_32(s_tm, [&](int c0, uint32_t (&v)[32]) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    float e[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float s = __uint_as_float(v[j + i]);
                        const float x = CAP ? fmaf(-score.cap2, rcp(ex2(s * score.k) + 1.0f), shift) : fmaf(s, score.k, shift);
                        e[i] = ex2(x);
                        if (decltype(masked)::value && c0 + j + i > seen) e[i] = 0.0f;
                    }
                    l0 += e[0];
                    l1 += e[1];
                    const uint32_t h = ptx::pack2(e[0], e[1]);
                    hi[j / 2] = h;
                    lo[j / 2] = ptx::pack2(e[0] - __uint_as_float(h << 16), e[1] - __uint_as_float(h & 0xffff0000u));
                }
                ptx::tmem_st16(s_tm + c0, hi);
                ptx::tmem_st16(s_tm + c0 + 16, lo);
            });
            };
            if (mask) weights(std::true_type{});
            else weights(std::false_type{});
            ptx::tmem_st_wait();
            // Not a tile ahead of the MMA thread: with three places the scores of tile t exist before the product of tile t - 2, and a
            // second arrival on p_full while that product still waits for its values would complete a phase that nobody has seen.
            if (t >= 2) ok &= ptx::mbar_wait_bounded(&sm.o_done[w], (uint32_t)(((t - 2) >> 1) & 1));
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&sm.p_full[w]);
        }
        // ---- both groups' halves: sums and references through shared memory, outputs in tensor memory ----
        const int own = w < tiles ? (tiles - 1 - w) / 2 : -1;  // this group's last use of its barriers
        if (own >= 0) ok &= ptx::mbar_wait_bounded(&sm.o_done[w], (uint32_t)(own & 1));
        ptx::tc_fence_after();
        sm.m[w][r] = m_ref;
        sm.l[w][r] = l0 + l1;
        ptx::tc_fence_before();
        ptx::named_bar_sync(1, kSoftmaxWarps * 32);
        ptx::tc_fence_after();
        const float m0 = sm.m[0][r], m1 = sm.m[1][r], m2 = fmaxf(m0, m1);
        float f0 = m0 == kNone ? 0.0f : ex2(m0 - m2), f1 = m1 == kNone ? 0.0f : ex2(m1 - m2);
        const float m_nat = m2 * kLn2;
        float den = sm.l[0][r] * f0 + sm.l[1][r] * f1, f = 1.0f;
        if (a.sink) {
            const float sk = a.sink[head], m = fmaxf(m_nat, sk);
            f = expf(m_nat - m);
            den = den * f + expf(sk - m);
        }
        f /= den;
        const int64_t row = (int64_t)b * a.q_rows + q0 + r;
        if (LATENT && lt.gate && r < rows) f /= 1.0f + expf(-lt.gate[row * lt.gate_ld + head]);
        f0 *= f;
        f1 *= f;
        const int dv = a.dv;
        const bool whole = dv % 8 == 0;  // groups of eight outputs are 16-byte pieces of the tiled layout
        for (int ch = w; ch < nv; ch += 2) {
            uint32_t o0[16], o1[16];
            ptx::tmem_ld16(o_tm + ch * 16, o0);
            if (tiles > 1) ptx::tmem_ld16(o_tm + o_cols + ch * 16, o1);
            ptx::tmem_ld_wait();
            float y[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                y[j] = __uint_as_float(o0[j]) * f0;
                if (tiles > 1) y[j] = fmaf(__uint_as_float(o1[j]), f1, y[j]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = ch * 16 + h * 8, col = head * dv + c;
                if (r >= rows) {
                    // (the warp's tensor-memory loads need all of its lanes)
                } else if (whole) {
                    if (c < dv)
                        *reinterpret_cast<uint4*>(out.tiles + dense_off(row, col, out.m_pad)) =
                            make_uint4(ptx::pack2(y[8 * h], y[8 * h + 1]), ptx::pack2(y[8 * h + 2], y[8 * h + 3]), ptx::pack2(y[8 * h + 4], y[8 * h + 5]), ptx::pack2(y[8 * h + 6], y[8 * h + 7]));
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c + j < dv) *reinterpret_cast<__nv_bfloat16*>(out.tiles + dense_off(row, col + j, out.m_pad)) = __float2bfloat16_rn(y[8 * h + j]);
                }
            }
            __syncwarp();
        }
    }
    if (!ok && a.err) atomicExch(a.err, kErrFlashTimeout);
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) ptx::tmem_dealloc(tmem, 512);
}

// What a launch needs of the kernel, once per device.
template <bool LATENT, bool CAP>
cudaError_t flash_ready() {
    static PerDeviceOnce once;
    return once.run([] {
        cudaError_t e = cudaFuncSetAttribute(attn_flash_kernel<LATENT, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFlashSmemMost);
        // (a share beyond what the launch gives the CTA would be waited for without end)
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, attn_flash_kernel<LATENT, CAP>);
        if (e != cudaSuccess) (void)cudaGetLastError();  // (answered by the caller, not by the next launch)
        return e == cudaSuccess && fa.numRegs * kFlashThreads < kRegsShares ? cudaErrorLaunchOutOfResources : e;
    });
}
template <bool LATENT, bool CAP>
cudaError_t flash_launch(const DenseAttn& a, const LatentTile& lt, const ActOut& out, cudaStream_t s) {
    const cudaError_t e = flash_ready<LATENT, CAP>();
    if (e != cudaSuccess) return e;
    const size_t smem = flash_bytes((a.kv.k_stride + 15) / 16, (a.kv.v_stride + 15) / 16) + sizeof(FlashSmem);
    attn_flash_kernel<LATENT, CAP><<<dim3((unsigned)a.heads, (unsigned)((a.q_rows + kFlashQ - 1) / kFlashQ), (unsigned)a.batch), kFlashThreads, smem, s>>>(a, lt, out);
    return cudaGetLastError();
}

}  // namespace

// Heads whose operands fit shared memory (three tiles of keys' width, two of values') and whose two accumulators fit tensor
// memory; positive scales (the softmax takes the largest raw score for the largest score); a build whose kernel has the
// registers that its warpgroups share out.
bool attn_flash_fits(const DenseAttn& a, bool latent) {
    if (a.kv.f32 || a.kv.k_stride > kFlashMaxK || a.kv.v_stride > kFlashMaxV || !(a.scale > 0.0f)) return false;
    const bool cap = a.softcap > 0.0f;
    return (latent ? (cap ? flash_ready<true, true>() : flash_ready<true, false>()) : (cap ? flash_ready<false, true>() : flash_ready<false, false>())) == cudaSuccess;
}

cudaError_t launch_attn_flash(const DenseAttn& a, const LatentTile* lt, const ActOut& out, cudaStream_t s) {
    if (!attn_flash_fits(a, lt != nullptr) || !a.q_bf16 || !out.tiles) return cudaErrorInvalidValue;
    const bool cap = a.softcap > 0.0f;
    if (lt) return cap ? flash_launch<true, true>(a, *lt, out, s) : flash_launch<true, false>(a, *lt, out, s);
    return cap ? flash_launch<false, true>(a, LatentTile(), out, s) : flash_launch<false, false>(a, LatentTile(), out, s);
}

}  // namespace bt

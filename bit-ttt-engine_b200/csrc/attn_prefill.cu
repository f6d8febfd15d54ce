// Causal attention of many new tokens per sequence over the Q8 KV cache (layers/attention.rs:198-217 on a prompt) on the
// tcgen05 integer tensor cores, with the arithmetic of the decode kernel: a rotated query value is S * Q / 2^27 with four
// signed 7-bit digits, a weight p * v_scale is B * U / 2^32 with four unsigned bytes and B = the power of two above the largest
// value scale of 512 positions, all digit sums are exact int32 accumulators, and the softmax runs in f32.  The scores are
// the decode kernel's bit by bit; the sums are taken in another order.
//
// Two kernels.  prefill_rows_kernel turns the q | k | v rows of the new tokens into what the attention reads: keys (rotated)
// and values into the cache as the append of a single token does, queries (rotated) into their digits, in place - a head's
// hd floats become its four rows of hd digit bytes.  prefill_attn_kernel is a persistent kernel, a CTA per SM: an item is
// (sequence, KV head, 64 query vectors = 64 / rep positions x rep heads of the group) and walks the key positions in tiles
// of 128.  Everything is transposed, so that a TMEM lane is a POSITION and the digits are columns:
//   S^T [128 positions, 4 x 32] = K tile . digits^T     A = key rows as they lie in the cache (K-major), B = digit rows
//   O^T [128 dims, 4 x 32]     += V tile^T . U          A = value rows as they lie in the cache (MN-major), B = weight words
// A lane then holds the four digit sums of a score side by side and joins them without any exchange, a position's two
// scales are a lane's own registers, and a weight word goes to shared memory as it is: its bytes are the four digit columns
// of the MN-major B operand.  Cache bytes only lose their offset of 128 on the way to shared memory (xor 0x80).
// The 64 query vectors are two groups of 32 with eight softmax warps and an MMA warp each, so that one group's softmax runs
// under the other's MMAs; four loader warps fill a ring of three K | V tiles.
// Softmax reference of a vector: the largest score so far, or one that a score exceeds by less than what B leaves free above
// its position's value scale (a weight is below B then, and U below 2^32).  While it holds, the integer accumulators run on from tile to
// tile; where a score breaks it, that vector's four columns are read out, joined into f32 sums in shared memory and
// rescaled, and of all vectors where B changes.
//
// mma.sync form -> this (a layer's launch): 8B shape, 2048 tokens 868 -> 204 us, 16 x 128 tokens 300 -> 56; 1B shape (heads of
// 64), 4 x 511 tokens 298 -> 73 us, 16 x 128 tokens 231 -> 50; 2 tokens 10.7 -> 10.3; 16 tokens after 2000 51.9 -> 48.5.  Bound by the
// instructions of the softmax warps (8B shape, 2048 tokens: issue slots 63 % busy, tensor pipe 17 %) and the latency of a
// group's chain scores - vote - weights - products.  Random scores ask for moves of references in most tiles; a weight word
// with two bits left free for scores above the reference needed hardly any (184 us), but a weight then had 30 bits.  Room by
// position instead of by the largest scale of the bound's tiles, and f32 sums that start at zero instead of being selected: 227 -> 206.
// With four softmax warps to a group (32 vectors a thread) the short items of heads of 64 took 1.5 times as long; scores
// and weights through integer conversion instructions 1.1 times; columns read out by fours of vectors 1.05 times, unrolled
// 1.2; warps without dims (heads of 64) sent past the read-outs 1.08.
#include <cfloat>
#include <type_traits>

#include "bt_common.cuh"
#include "bt_model.cuh"
#include "bt_ptx.cuh"

namespace bt {

namespace {

constexpr int kTilePos = 128;            // positions of a tile = TMEM lanes
constexpr int kGroupVec = 32;            // query vectors of a group
constexpr int kCols = 4 * kGroupVec;     // digit columns = N of the MMAs
constexpr int kStages = 3;
constexpr int kChunk = kTilePos * 16 + 16;   // bytes between the 16-byte column chunks of an operand tile (the odd 16: a row's
                                             // chunks, written by neighbouring lanes, fall into different banks)
constexpr int kOpBytes = 8 * kChunk;         // an operand tile of up to 128 columns (bytes)
constexpr int kPChunk = kTilePos * 16;       // the same of the weight words, whose writers are neighbouring positions
constexpr int kPBytes = 8 * kPChunk;
constexpr int kSoftWarps = 16, kLoadWarps = 4;
constexpr int kHalfVec = kGroupVec / 2, kHalfThreads = 128;
constexpr int kThreads = (kSoftWarps + kLoadWarps + 4) * 32;  // + an MMA warp per group, two idle: the roles are whole warpgroups
constexpr int kRegsSoft = 96, kRegsLoad = 56, kRegsMma = 40;
constexpr int kMaxDim = 128;
constexpr int kBoundTiles = 4;           // tiles of a weight bound
constexpr int kMaxRun = 256;             // tiles between two read-outs at most: 256 * 128 positions * 255 * 128 < 2^31
// Integers become floats without a conversion (16 a clock and SM, as the exponential): an integer below 2^22 added to the bit
// pattern of kMagic is the pattern of kMagic plus that integer.  The score accumulators start at the pattern, so that the
// MMAs leave floats; kMagicHi takes it out of a digit and, 128 times smaller, out of the digit below in the same addition.
constexpr float kMagic = 12582912.0f;               // 1.5 * 2^23
constexpr uint32_t kMagicBits = 0x4b400000u;
constexpr float kMagicHi = kMagic + kMagic / 128;
constexpr float kMagicWord = kMagic + 0xb4c0;       // 0xb4c0 + 0x4b40 = 0x10000: the patterns of a word's two halves cancel
constexpr unsigned kErrPrefillAttn = 0x50464154u;  // 'PFAT'

struct Smem {
    alignas(128) uint8_t kv[kStages][2][kOpBytes];     // [stage][keys | values]
    alignas(128) uint8_t q[2][kOpBytes];               // query digits of a group
    alignas(128) uint8_t u[2][kPBytes];                // weight words of a group's tile
    alignas(16) float osum[2][kGroupVec][kMaxDim];     // what has been read out of the accumulators
    alignas(16) float cq[2][kGroupVec];                // S / 2^27 times the score scaling
    alignas(16) float mref[2][kGroupVec];              // reference of the weights
    alignas(16) float fac[2][kGroupVec];               // e^(old - new reference) of a move; at the end the denominators
    alignas(16) int seen[2][kGroupVec];                // last position a vector sees
    alignas(16) int at[2][2][kGroupVec];               // [item & 1]: where its output goes (-1: nowhere)
    float wred[2][4][kGroupVec];                       // per warp: maxima of a tile, sums at the end
    uint32_t moved[2][2];                              // per half: the vectors whose reference moves
    alignas(16) float wv[2][2][4];                                 // per half and warp: largest value scale of a bound's tiles
    uint64_t full[kStages], empty[kStages];
    uint64_t q_full[2], q_empty[2], s_full[2], s_empty[2], p_full[2], pv_done[2];
    uint32_t tmem;
};

// kind::i8, D = s32, M = N = 128.  a_signed / b_signed: s8 or u8 operands; mn: both operands MN-major instead of K-major.
__device__ __forceinline__ constexpr uint32_t instr_desc(bool a_signed, bool b_signed, bool mn) {
    return (2u << 4) | (uint32_t)a_signed << 7 | (uint32_t)b_signed << 10 | (mn ? 3u << 15 : 0u) | (uint32_t)(kCols >> 3) << 17 | (uint32_t)(kTilePos >> 4) << 24;
}

__device__ __forceinline__ bool bar_or(int id, int threads, bool flag) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\t"
        "barrier.cta.red.or.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r) : "r"(id), "r"(threads), "r"((uint32_t)flag) : "memory");
    return r != 0;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
// the loads into v are complete (v is named, so that no use of it is moved before the wait)
__device__ __forceinline__ void ld_wait16(uint32_t (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                   "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
                 :: "memory");
}
// four consecutive columns of this thread's tensor-memory lane, which are zero afterwards
__device__ __forceinline__ void tmem_take4(uint32_t taddr, uint32_t (&v)[4]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n\t"
        "tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%5, %5, %5, %5};"
        : "=&r"(v[0]), "=&r"(v[1]), "=&r"(v[2]), "=&r"(v[3]) : "r"(taddr), "r"(0) : "memory");
}
// An item of the persistent loop: the heaviest query blocks first, dealt to the CTAs forwards and backwards in turn.
struct Item {
    int b, kvh, q0, p, tiles, t_len;
};
struct Items {
    const PrefillAttnArgs& a;
    int pairs, blocks, per;  // per = new tokens of an item
    __device__ Items(const PrefillAttnArgs& args) : a(args), pairs(args.batch * args.n_kv), per(2 * kGroupVec >> args.rep_log) {
        blocks = (a.q_rows + per - 1) / per;
    }
    __device__ bool get(int round, Item* it) const {
        const int g = (int)gridDim.x, i = round * g + (round & 1 ? g - 1 - (int)blockIdx.x : (int)blockIdx.x);
        if (i >= pairs * blocks) return false;
        const int pair = i % pairs;
        it->q0 = (blocks - 1 - i / pairs) * per;
        it->b = pair / a.n_kv;
        it->kvh = pair % a.n_kv;
        it->p = a.pos[it->b];
        it->t_len = it->p + min(it->q0 + per, a.q_rows);
        it->tiles = (it->t_len + kTilePos - 1) / kTilePos;
        return true;
    }
};

template <int HD>
__global__ void __launch_bounds__(kThreads, 1) prefill_attn_kernel(PrefillAttnArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) { ptx::mbar_init(&sm.full[i], kLoadWarps * 32); ptx::mbar_init(&sm.empty[i], 2); }
        for (int g = 0; g < 2; ++g) {
            ptx::mbar_init(&sm.q_full[g], kLoadWarps * 32);
            ptx::mbar_init(&sm.q_empty[g], 1);
            ptx::mbar_init(&sm.s_full[g], 1);
            ptx::mbar_init(&sm.s_empty[g], kSoftWarps / 2);
            ptx::mbar_init(&sm.p_full[g], kSoftWarps / 2);
            ptx::mbar_init(&sm.pv_done[g], 1);
        }
        ptx::mbar_fence_init();
    }
    if (warp == kSoftWarps + kLoadWarps) {
        ptx::tmem_alloc(&sm.tmem, 512);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = sm.tmem;  // S of group 0 | S of group 1 | O of group 0 | O of group 1, kCols columns each
    const Items items(a);
    bool ok = true;
    // Completion n (0, 1, ...) of a barrier; after a wait that gave up, nothing waits any more.  Relaxed: what a barrier of this
    // kernel hands over is read by the tensor core (its writers have fenced it) or lies in tensor memory (ordered by the
    // tcgen05 fences), never read by loads of the thread that waits.
    auto wait = [&](uint64_t* bar, int n) {
        if (ok) ok = ptx::mbar_spin_relaxed(bar, (uint32_t)(n & 1));
    };

    if (warp < kSoftWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoft));
        // ---------------- softmax of group g: thread = position (scores, weights) or dim (outputs) r, half of the vectors ----------------
        const int g = warp >> 3, w4 = warp & 3, r = 32 * w4 + lane, half = warp >> 2 & 1, h0 = half * kHalfVec, th = tid & (kHalfThreads - 1), bar_id = 1 + (warp >> 2);
        const int own = h0 + th;  // th < kHalfVec: the vector this thread looks after
        const uint32_t s_addr = tmem + ((uint32_t)(32 * w4) << 16) + g * kCols + 4 * h0, o_addr = s_addr + 2 * kCols;
        const int per_group = kGroupVec >> a.rep_log;
        uint32_t magic[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) magic[i] = kMagicBits;
#pragma unroll
        for (int c = 0; c < kHalfVec / 4; ++c) {
            ptx::tmem_st16(s_addr + 16 * c, magic);
            ptx::tmem_st16(o_addr + 16 * c, {});
        }
        ptx::tmem_st_wait();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sm.s_empty[g]);
        int n = 0;  // tiles of all items so far
        Item it = {};
        // what the first tile of an item needs from global memory, requested before the item in front is finished
        // (a value scale that is no number or negative counts as zero, as it does in the decode kernel)
        float ks_next = 0.0f, vs_next = 0.0f, q_scale = 0.0f;
        auto value_scale = [&](const float* vs, int at, int t_len) { return at < t_len ? fmaxf(vs[at], 0.0f) : 0.0f; };
        auto prefetch = [&]() {
            const int64_t row = ((int64_t)it.b * a.n_kv + it.kvh) * a.cache.max_seq;
            ks_next = r < it.t_len ? a.cache.k_s[row + r] : 0.0f;
            vs_next = value_scale(a.cache.v_s + row, r, it.t_len);
            if (th < kHalfVec) {
                const int tok = min(it.q0 + g * per_group + (own >> a.rep_log), a.q_rows - 1);  // (beyond the last token: the last again, not stored)
                q_scale = a.qscale[((int64_t)it.b * a.q_rows + tok) * a.n_heads + (it.kvh << a.rep_log) + (own & ((1 << a.rep_log) - 1))];
            }
        };
        bool more = items.get(0, &it);
        if (more) prefetch();
        for (int round = 0; more; ++round) {
            const int64_t row_base = ((int64_t)it.b * a.n_kv + it.kvh) * a.cache.max_seq;
            const float *ks = a.cache.k_s + row_base, *vs = a.cache.v_s + row_base;
            const int first = it.q0 + g * per_group;  // the group's first new token
            const int first_seen = it.p + min(first, a.q_rows - 1), tiles = it.tiles, t_len = it.t_len;
            if (th < kHalfVec) {
                const int tok = first + (own >> a.rep_log);
                sm.cq[g][own] = __fmul_rn(q_scale, a.scaling);
                sm.seen[g][own] = it.p + min(tok, a.q_rows - 1);
                sm.mref[g][own] = -FLT_MAX;
                sm.at[round & 1][g][own] = tok < a.q_rows ? (tok * a.n_heads + (it.kvh << a.rep_log) + (own & ((1 << a.rep_log) - 1))) * HD : -1;
            }
            float l[kHalfVec], s[kHalfVec];
#pragma unroll
            for (int v = 0; v < kHalfVec; ++v) {
                l[v] = 0.0f;
                sm.osum[g][h0 + v][r] = 0.0f;
            }
            uint32_t ex = 0, ex_new = 0;  // exponent of the weight bound, of these tiles and of the next kBoundTiles
            float up = 0.0f, down = 0.0f, room = 0.0f;  // room: how far a score may exceed its reference
            ptx::named_bar_sync(bar_id, kHalfThreads);
            // of vector v, whose four digit columns are b: the accumulator as f32, joined with what was read out before
            auto joined = [&](const uint32_t* b, int v) {
                const long long sum = (long long)(int)b[3] * (1 << 24) + ((long long)(int)b[2] * (1 << 16) + ((long long)(int)b[1] * (1 << 8) + (int)b[0]));
                return fmaf(__ll2float_rn(sum), down, sm.osum[g][h0 + v][r]);
            };
            // lane v % 16 ends with the warp's join of vector h0 + v (x is consumed)
            auto across = [&](float (&x)[kHalfVec], auto join) {
#pragma unroll
                for (int o = kHalfVec / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int v = 0; v < o; ++v) {
                        const float give = lane & o ? x[v] : x[v + o], keep = lane & o ? x[v + o] : x[v];
                        x[v] = join(keep, __shfl_xor_sync(0xffffffffu, give, o));
                    }
                x[0] = join(x[0], __shfl_xor_sync(0xffffffffu, x[0], 16));
                if (lane < kHalfVec) sm.wred[g][w4][h0 + lane] = x[0];
            };
            for (int t = 0; t < tiles; ++t, ++n) {
                const float k_scale = ks_next, v_scale = vs_next;
                const int at = t * kTilePos + r;
                // The value scales of the next bound's tiles are looked at in the tile before its first one (of the first bound: in
                // the first), so that the bound is known when that tile's scores are compared with their reference.
                const bool look = t == 0 || (t % kBoundTiles == kBoundTiles - 1 && t + 1 < tiles);
                float v_look[kBoundTiles] = {};
                if (look) {
                    const int from = at + (t > 0 ? kTilePos : 0);
#pragma unroll
                    for (int i = 0; i < kBoundTiles; ++i) v_look[i] = value_scale(vs, from + i * kTilePos, t_len);
                }
                if (t + 1 < tiles) {
                    ks_next = at + kTilePos < t_len ? ks[at + kTilePos] : 0.0f;
                    vs_next = value_scale(vs, at + kTilePos, t_len);
                }
                wait(&sm.s_full[g], n);
                ptx::tc_fence_after();
                // How far this position's scores may exceed their references: its weights are below the bound while the exponential
                // is below bound / scale (the bound of this tile, already; the first tile sets the references).  2^-16 is more than
                // the errors of the logarithm and the exponential.
                const float share = __fmul_rn(v_scale, __uint_as_float((270 - ex_new) << 23));  // scale / bound * 2^16
                const float room_here = t > 0 ? fmaxf(room, fminf(11.0903549f - __logf(share) - 1.0f / 65536.0f, 0.69f)) : 0.0f;
                const float v_most = fmaxf(fmaxf(v_look[0], v_look[1]), fmaxf(v_look[2], v_look[3]));
                bool over = false;  // some score is too far above its reference
                auto scores = [&](auto masked_tag) {
                    constexpr bool kMasked = decltype(masked_tag)::value;
                    uint32_t d[2][16];
                    ptx::tmem_ld16(s_addr, d[0]);
#pragma unroll
                    for (int c = 0; c < kHalfVec / 4; ++c) {
                        ld_wait16(d[c & 1]);
                        if (c + 1 < kHalfVec / 4) ptx::tmem_ld16(s_addr + 16 * (c + 1), d[(c + 1) & 1]);
                        ptx::tmem_st16(s_addr + 16 * c, magic);  // (the loads of these columns are complete)
                        const float4 cq = *reinterpret_cast<const float4*>(&sm.cq[g][h0 + 4 * c]), mr = *reinterpret_cast<const float4*>(&sm.mref[g][h0 + 4 * c]);
                        const float cqv[4] = {cq.x, cq.y, cq.z, cq.w}, mrv[4] = {mr.x, mr.y, mr.z, mr.w};
                        int4 last = make_int4(0, 0, 0, 0);
                        if (kMasked) last = *reinterpret_cast<const int4*>(&sm.seen[g][h0 + 4 * c]);
                        const int lastv[4] = {last.x, last.y, last.z, last.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t* b = &d[c & 1][4 * i];
                            const float hi = fmaf(__fsub_rn(__uint_as_float(b[0]), kMagicHi), 128.0f, __uint_as_float(b[1]));
                            const float lo = fmaf(__fsub_rn(__uint_as_float(b[2]), kMagicHi), 128.0f, __uint_as_float(b[3]));
                            float x = __fmul_rn(__fmul_rn(fmaf(hi, 16384.0f, lo), k_scale), cqv[i]);
                            if (kMasked && at > lastv[i]) x = -INFINITY;
                            s[4 * c + i] = x;
                            over |= __fsub_rn(x, mrv[i]) > room_here;
                        }
                    }
                };
                // (a tile whose last position the group's first query may see needs no mask)
                if (t * kTilePos + kTilePos - 1 <= first_seen) scores(std::false_type{});
                else scores(std::true_type{});
                ptx::tmem_st_wait();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm.s_empty[g]);
                if (__any_sync(0xffffffffu, over)) {
                    float m[kHalfVec];
#pragma unroll
                    for (int v = 0; v < kHalfVec; ++v) m[v] = s[v];
                    across(m, [](float x, float y) { return fmaxf(x, y); });
                } else if (lane < kHalfVec) {
                    sm.wred[g][w4][h0 + lane] = -FLT_MAX;
                }
                if (look) {
                    const unsigned vm = __reduce_max_sync(0xffffffffu, __float_as_uint(v_most));
                    if (lane == 0) sm.wv[g][half][w4] = __uint_as_float(vm);
                }
                const bool move = bar_or(bar_id, kHalfThreads, over);
                if (n > 0) {
                    wait(&sm.pv_done[g], n - 1);  // the weight words are free, the accumulators hold the tiles before
                    ptx::tc_fence_after();
                }
                const bool new_bound = t % kBoundTiles == 0, all = (new_bound && ex_new != ex) || t % kMaxRun == 0;
                const float room_now = room;
                if (look) {
                    // The power of two above the largest value scale of these tiles, and 2^-19 more, so that a weight is below 2^32
                    // whatever the last bits of its exponential (kept where the bound and 2^-32 of it are floats).  What that
                    // power leaves free is room for scores above the reference.
                    const float4 v4 = *reinterpret_cast<const float4*>(sm.wv[g][half]);
                    const float big = fmaxf(fmaxf(v4.x, v4.y), fmaxf(v4.z, v4.w));
                    const uint32_t bits = __float_as_uint(fmaf(big, 1.0f / 524288.0f, big));
                    ex_new = min(max((bits >> 23) + 1, 33u), 254u);
                    room = (bits >> 23) < 254u ? fmaxf(-logf(__uint_as_float((bits & 0x7fffffu) | 126u << 23)) - 1.0f / 262144.0f, 0.0f) : 0.0f;
                }
                if (move || (all && t > 0)) {
                    if (move) {
                        if (th < kHalfVec) {
                            const float old = sm.mref[g][own], most = fmaxf(fmaxf(sm.wred[g][0][own], sm.wred[g][1][own]), fmaxf(sm.wred[g][2][own], sm.wred[g][3][own]));
                            const bool moves = __fsub_rn(most, old) > room_now;
                            const uint32_t moved = __ballot_sync(0xffffu, moves);
                            if (th == 0) sm.moved[g][half] = t > 0 ? moved : 0u;
                            sm.fac[g][own] = moves ? expf(__fsub_rn(old, most)) : 1.0f;
                            if (moves) sm.mref[g][own] = most;
                        }
                        ptx::named_bar_sync(bar_id, kHalfThreads);
#pragma unroll
                        for (int c = 0; c < kHalfVec / 4; ++c) {
                            const float4 f = *reinterpret_cast<const float4*>(&sm.fac[g][h0 + 4 * c]);
                            l[4 * c] *= f.x; l[4 * c + 1] *= f.y; l[4 * c + 2] *= f.z; l[4 * c + 3] *= f.w;
                        }
                    }
                    // read out the vectors whose reference has moved (of a new bound all); their columns are zero afterwards.  (Not
                    // unrolled: this code is run rarely and together, and the rest of the loop has to stay in the instruction cache.)
                    const uint32_t which = all && t > 0 ? (1u << kHalfVec) - 1 : sm.moved[g][half];
#pragma unroll 1
                    for (uint32_t rest = which; rest; rest &= rest - 1) {
                        const int v = __ffs(rest) - 1;
                        uint32_t d[4];
                        tmem_take4(o_addr + 4 * v, d);
                        sm.osum[g][h0 + v][r] = joined(d, v) * (move ? sm.fac[g][h0 + v] : 1.0f);
                    }
                    ptx::tmem_st_wait();
                }
                if (new_bound) {
                    ex = ex_new;
                    up = __uint_as_float((270 - ex) << 23);   // 2^16 / bound
                    down = __uint_as_float((ex - 32) << 23);  // bound / 2^32
                }
                const float w_scale = fminf(__fmul_rn(v_scale, up), 65535.9375f);  // (smaller already, but for scales beyond the last bound)
                uint8_t* words = sm.u[g] + h0 / 4 * kPChunk + r * 16;
#pragma unroll
                for (int c = 0; c < kHalfVec / 4; ++c) {
                    const float4 mr = *reinterpret_cast<const float4*>(&sm.mref[g][h0 + 4 * c]);
                    const float mrv[4] = {mr.x, mr.y, mr.z, mr.w};
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float e = expf(__fsub_rn(s[4 * c + i], mrv[i]));
                        l[4 * c + i] += e;
                        const float upper = fmaf(e, w_scale, kMagicWord);  // the word's upper half, rounded; what is left of it (signed) in 2^-16
                        const float rest = fmaf(e, w_scale, -__fsub_rn(upper, kMagicWord));
                        w[i] = (__float_as_uint(upper) << 16) + __float_as_uint(fmaf(rest, 65536.0f, kMagic));
                    }
                    *reinterpret_cast<uint4*>(words + c * kPChunk) = make_uint4(w[0], w[1], w[2], w[3]);
                }
                ptx::fence_async_smem();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm.p_full[g]);
            }
            float* out = a.out + (int64_t)it.b * a.q_rows * a.n_heads * HD + r;
            more = items.get(round + 1, &it);
            if (more) prefetch();
            across(l, [](float x, float y) { return x + y; });
            ptx::named_bar_sync(bar_id, kHalfThreads);
            if (th < kHalfVec) sm.fac[g][own] = (sm.wred[g][0][own] + sm.wred[g][1][own]) + (sm.wred[g][2][own] + sm.wred[g][3][own]);
            wait(&sm.pv_done[g], n - 1);
            ptx::tc_fence_after();
            ptx::named_bar_sync(bar_id, kHalfThreads);
            uint32_t d[2][16];
            ptx::tmem_ld16(o_addr, d[0]);
#pragma unroll
            for (int c = 0; c < kHalfVec / 4; ++c) {
                ld_wait16(d[c & 1]);
                if (c + 1 < kHalfVec / 4) ptx::tmem_ld16(o_addr + 16 * (c + 1), d[(c + 1) & 1]);
                ptx::tmem_st16(o_addr + 16 * c, {});
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int v = 4 * c + i, to = sm.at[round & 1][g][h0 + v];
                    const float o = joined(&d[c & 1][4 * i], v);
                    if (to >= 0 && r < HD) out[to] = __fdiv_rn(o, sm.fac[g][h0 + v]);
                }
            }
            ptx::tmem_st_wait();
            ptx::tc_fence_before();
        }
    } else if (warp < kSoftWarps + kLoadWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsLoad));
        // ---------------- loader warps ----------------
        constexpr int P16 = HD / 16, kPieces = kTilePos * P16 / (kLoadWarps * 32);  // 16-byte pieces per row; per thread and tile
        const int lt = tid - kSoftWarps * 32;
        const int64_t q_stride = (int64_t)(a.n_heads + 2 * a.n_kv) * HD * 4;  // bytes of a q | k | v row
        int n = 0;
        Item it;
        for (int round = 0; items.get(round, &it); ++round) {
            const int64_t row_base = ((int64_t)it.b * a.n_kv + it.kvh) * a.cache.max_seq;
            for (int t = 0; t < it.tiles; ++t, ++n) {
                const int st = n % kStages;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const uint8_t* src = (half ? a.cache.v_q : a.cache.k_q) + (row_base + (int64_t)t * kTilePos) * HD;
                    uint4 d[kPieces];
#pragma unroll
                    for (int k = 0; k < kPieces; ++k) {
                        const int i = lt + k * kLoadWarps * 32;
                        d[k] = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
                        if (t * kTilePos + i / P16 < it.t_len) d[k] = *reinterpret_cast<const uint4*>(src + (int64_t)i * 16);
                    }
                    if (half == 0 && n >= kStages) wait(&sm.empty[st], n / kStages - 1);
#pragma unroll
                    for (int k = 0; k < kPieces; ++k) {
                        const int i = lt + k * kLoadWarps * 32;
                        *reinterpret_cast<uint4*>(sm.kv[st][half] + (i % P16) * kChunk + (i / P16) * 16) =
                            make_uint4(d[k].x ^ 0x80808080u, d[k].y ^ 0x80808080u, d[k].z ^ 0x80808080u, d[k].w ^ 0x80808080u);
                    }
                }
                ptx::fence_async_smem();
                ptx::mbar_arrive(&sm.full[st]);
                if (t > 0) continue;
                // the queries after the first tile: their place is free once the item in front has issued its last scores
                for (int g = 0; g < 2; ++g) {
                    uint4 d[kPieces];
#pragma unroll
                    for (int k = 0; k < kPieces; ++k) {
                        const int i = lt + k * kLoadWarps * 32, col = i / P16, v = col >> 2;  // column 4 v + j = digit j of vector v
                        const int tok = min(it.q0 + (((g * kGroupVec) + v) >> a.rep_log), a.q_rows - 1), h = (it.kvh << a.rep_log) + (v & ((1 << a.rep_log) - 1));
                        d[k] = *reinterpret_cast<const uint4*>(a.qdig + ((int64_t)it.b * a.q_rows + tok) * q_stride + (int64_t)(4 * h + (col & 3)) * HD + (i % P16) * 16);
                    }
                    if (round > 0) wait(&sm.q_empty[g], round - 1);
#pragma unroll
                    for (int k = 0; k < kPieces; ++k) {
                        const int i = lt + k * kLoadWarps * 32;
                        *reinterpret_cast<uint4*>(sm.q[g] + (i % P16) * kChunk + (i / P16) * 16) = d[k];
                    }
                    ptx::fence_async_smem();
                    ptx::mbar_arrive(&sm.q_full[g]);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsMma));
        // ---------------- MMA warp of group g: the whole warp runs the loop, so that descriptors and addresses are uniform
        //                  registers; one elected thread issues ----------------
        if (warp < kSoftWarps + kLoadWarps + 2) {
            const int g = warp - kSoftWarps - kLoadWarps;
            constexpr uint32_t qk = instr_desc(true, true, false), pv = instr_desc(true, false, true);
            constexpr uint64_t kKStep = 2 * kChunk >> 4, kPosStep = 512 >> 4, kStageStep = 2 * kOpBytes >> 4;  // in a descriptor's address units
            const uint64_t q_desc = ptx::smem_desc(ptx::smem_u32(sm.q[g]), kChunk, 128), u_desc = ptx::smem_desc(ptx::smem_u32(sm.u[g]), 128, kPChunk);
            const uint64_t k_desc = ptx::smem_desc(ptx::smem_u32(sm.kv[0][0]), kChunk, 128), v_desc = ptx::smem_desc(ptx::smem_u32(sm.kv[0][1]), 128, kChunk);
            const uint32_t s_tmem = tmem + g * kCols, o_tmem = tmem + (2 + g) * kCols;
            auto values = [&](int m, int st) {  // O += V^T . U of tile m
                wait(&sm.p_full[g], m);
                ptx::tc_fence_after();
                const uint64_t vd = v_desc + st * kStageStep;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < kTilePos / 32; ++k) ptx::umma_i8(o_tmem, vd + k * kPosStep, u_desc + k * kPosStep, pv, 1u);
                    ptx::umma_commit(&sm.pv_done[g]);
                    ptx::umma_commit(&sm.empty[st]);
                }
                __syncwarp();
            };
            int n = 0, st = 0, before = 0, use = 0;  // tile, its stage, the stage of the tile before, uses of the stage
            Item it;
            for (int round = 0; items.get(round, &it); ++round) {
                for (int t = 0; t < it.tiles; ++t, ++n) {
                    wait(&sm.full[st], use);
                    if (t == 0) wait(&sm.q_full[g], round);
                    wait(&sm.s_empty[g], n);
                    ptx::tc_fence_after();
                    const uint64_t kd = k_desc + st * kStageStep;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < HD / 32; ++k) ptx::umma_i8(s_tmem, kd + k * kKStep, q_desc + k * kKStep, qk, 1u);
                        ptx::umma_commit(&sm.s_full[g]);
                        if (t + 1 == it.tiles) ptx::umma_commit(&sm.q_empty[g]);
                    }
                    __syncwarp();
                    if (t > 0) values(n - 1, before);
                    before = st;
                    if (++st == kStages) { st = 0; ++use; }
                }
                values(n - 1, before);
            }
        }
    }
    if (!ok) atomicExch(a.err, kErrPrefillAttn);
    __syncthreads();
    if (warp == kSoftWarps + kLoadWarps) ptx::tmem_dealloc(tmem, 512);
}

// A token per blockIdx.x; a vector of HD values (a query, key or value head) per W lanes, four outputs a lane.  Bound by its
// instructions: the exact divisions of the cache quantiser and the digit arithmetic.
template <int HD>
__global__ void __launch_bounds__(256) prefill_rows_kernel(KvCacheView cache, float* __restrict__ qkv, const int32_t* __restrict__ pos,
                                                           const float* __restrict__ rope_cos, const float* __restrict__ rope_sin,
                                                           int q_rows, int n_heads, int n_kv, float* __restrict__ qscale) {
    constexpr int W = HD <= 32 ? 8 : (HD <= 64 ? 16 : 32), half = HD / 2;
    const int slots = n_heads + 2 * n_kv, lane = threadIdx.x % W;
    const int64_t row = blockIdx.x;
    const int b = (int)blockIdx.x / q_rows, p = pos[b] + (int)blockIdx.x % q_rows;
    const int slot = ((int)blockIdx.y * (int)blockDim.x + (int)threadIdx.x) / W;
    const bool active = slot < slots && 4 * lane < HD;
    float* src = qkv + row * (int64_t)slots * HD + (int64_t)slot * HD;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (active) {
        const float4 own = *reinterpret_cast<const float4*>(src + 4 * lane);
        v[0] = own.x; v[1] = own.y; v[2] = own.z; v[3] = own.w;
        if (slot < n_heads + n_kv) {  // [x1 cos - x2 sin, x1 sin + x2 cos] (layers/attention.rs:79-83)
            const bool second = 4 * lane >= half;
            const int c = second ? 4 * lane - half : 4 * lane;
            const float4 oth = *reinterpret_cast<const float4*>(src + (second ? c : c + half));
            const float4 c4 = *reinterpret_cast<const float4*>(rope_cos + (int64_t)p * half + c), s4 = *reinterpret_cast<const float4*>(rope_sin + (int64_t)p * half + c);
            const float o[4] = {oth.x, oth.y, oth.z, oth.w}, cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                v[i] = second ? __fadd_rn(__fmul_rn(o[i], sn[i]), __fmul_rn(v[i], cs[i])) : __fsub_rn(__fmul_rn(v[i], cs[i]), __fmul_rn(o[i], sn[i]));
        }
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));  // (also: every lane has read its part of the row)
    if (!active) return;
    if (slot < n_heads) {
        // Q = round(q / S * 2^27), S = the power of two above max|q|; Q = ((d0 * 128 + d1) * 128 + d2) * 128 + d3, digits in [-64, 64]
        const int ex = max((int)(__float_as_uint(amax) >> 23) - 126, -90);  // amax < 2^ex (kept where 2^(27 - ex) is a float)
        const float up = __uint_as_float((uint32_t)(154 - ex) << 23);
        uint32_t d[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int Q = __float2int_rn(__fmul_rn(v[i], up));
            const int d3 = ((Q + 64) & 127) - 64; Q = (Q - d3) >> 7;
            const int d2 = ((Q + 64) & 127) - 64; Q = (Q - d2) >> 7;
            const int d1 = ((Q + 64) & 127) - 64; Q = (Q - d1) >> 7;
            d[0] |= (uint32_t)(Q & 255) << (8 * i);
            d[1] |= (uint32_t)(d1 & 255) << (8 * i);
            d[2] |= (uint32_t)(d2 & 255) << (8 * i);
            d[3] |= (uint32_t)(d3 & 255) << (8 * i);
        }
        uint8_t* dst = reinterpret_cast<uint8_t*>(src);
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint32_t*>(dst + j * HD + 4 * lane) = d[j];
        if (lane == 0) qscale[row * n_heads + slot] = __uint_as_float((uint32_t)(100 + ex) << 23);
        return;
    }
    if (p < 0 || p >= cache.max_seq) return;
    // quantize_q8 (layers/kv_cache.rs:95-119): s = max|x| / 127, u8(round(x / s) + 128)
    const bool value = slot >= n_heads + n_kv;
    const int64_t r = ((int64_t)b * n_kv + (slot - n_heads - (value ? n_kv : 0))) * cache.max_seq + p;
    const float s = __fdiv_rn(amax, 127.0f);
    uint32_t w = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float q = s > 0.0f ? roundf(__fdiv_rn(v[i], s)) : 0.0f;
        w |= (uint32_t)(uint8_t)fminf(fmaxf(q + 128.0f, 0.0f), 255.0f) << (8 * i);
    }
    *reinterpret_cast<uint32_t*>((value ? cache.v_q : cache.k_q) + r * HD + 4 * lane) = w;
    if (lane == 0) (value ? cache.v_s : cache.k_s)[r] = s;
}

template <int HD>
cudaError_t launch_attn_hd(const PrefillAttnArgs& a, cudaStream_t stream) {
    static PerDeviceOnce once;
    cudaError_t e = once.run([] {
        // the register shares the warpgroups ask for must fit what the launch gives the CTA, or the asking waits for ever
        cudaFuncAttributes fa;
        cudaError_t e2 = cudaFuncGetAttributes(&fa, prefill_attn_kernel<HD>);
        if (e2 == cudaSuccess && fa.numRegs * kThreads < 128 * (kSoftWarps / 4 * kRegsSoft + kRegsLoad + kRegsMma)) e2 = cudaErrorLaunchOutOfResources;
        return e2 == cudaSuccess ? cudaFuncSetAttribute(prefill_attn_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)) : e2;
    });
    if (e != cudaSuccess) return e;
    const int per = 2 * kGroupVec >> a.rep_log;
    const int64_t n = (int64_t)a.batch * a.n_kv * ((a.q_rows + per - 1) / per);
    if (n > (1 << 30) || (int64_t)a.q_rows * a.n_heads * HD >= (1ll << 31)) return cudaErrorInvalidValue;
    prefill_attn_kernel<HD><<<(unsigned)(n < a.sm_count ? n : a.sm_count), kThreads, sizeof(Smem), stream>>>(a);
    return cudaGetLastError();
}

template <int HD>
cudaError_t launch_rows_hd(const KvCacheView& cache, float* qkv, const int32_t* pos, const float* rope_cos, const float* rope_sin, int batch,
                           int q_rows, int n_heads, int n_kv, float* qscale, cudaStream_t stream) {
    if ((int64_t)batch * q_rows > (1 << 30)) return cudaErrorInvalidValue;
    constexpr int W = HD <= 32 ? 8 : (HD <= 64 ? 16 : 32);
    const dim3 grid((unsigned)(batch * q_rows), (unsigned)(((n_heads + 2 * n_kv) * W + 255) / 256));
    prefill_rows_kernel<HD><<<grid, 256, 0, stream>>>(cache, qkv, pos, rope_cos, rope_sin, q_rows, n_heads, n_kv, qscale);
    return cudaGetLastError();
}

static_assert(sizeof(Smem) <= 227 * 1024, "shared memory");

}  // namespace

cudaError_t launch_prefill_attn(const PrefillAttnArgs& a, cudaStream_t stream) {
    if (a.rep_log < 0 || a.rep_log > 3 || a.n_heads != a.n_kv << a.rep_log || a.q_rows < 1 || a.batch < 1) return cudaErrorInvalidValue;
    switch (a.head_dim) {
        case 32: return launch_attn_hd<32>(a, stream);
        case 64: return launch_attn_hd<64>(a, stream);
        case 96: return launch_attn_hd<96>(a, stream);
        case 128: return launch_attn_hd<128>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_prefill_rows(const KvCacheView& cache, float* qkv, const int32_t* pos, const float* rope_cos, const float* rope_sin, int batch,
                                int q_rows, int n_heads, int n_kv, int hd, float* qscale, cudaStream_t stream) {
    switch (hd) {
        case 32: return launch_rows_hd<32>(cache, qkv, pos, rope_cos, rope_sin, batch, q_rows, n_heads, n_kv, qscale, stream);
        case 64: return launch_rows_hd<64>(cache, qkv, pos, rope_cos, rope_sin, batch, q_rows, n_heads, n_kv, qscale, stream);
        case 96: return launch_rows_hd<96>(cache, qkv, pos, rope_cos, rope_sin, batch, q_rows, n_heads, n_kv, qscale, stream);
        case 128: return launch_rows_hd<128>(cache, qkv, pos, rope_cos, rope_sin, batch, q_rows, n_heads, n_kv, qscale, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bt

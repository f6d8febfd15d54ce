// Batched / prefill ternary product on the 5th-generation tensor cores (tcgen05, TMEM):
//   acc[n, m] = sum_k t[n, k] * q[m, k]   for M > 8 tokens.
// Stands in for BitLinearCpu::forward / BitLinearCuda::forward (kernels/cpu.rs:17-127,
// kernels/cuda.rs:21-47) at batch and prefill sizes, where the reference runs a dense f32 GEMM
// on a host-unpacked weight.
//
// Roles inside one CTA (1 per SM, persistent over work units of RS x 128 weight rows x NT tokens x a k range;
// the RS = 1 or 2 row sets of a unit share every activation block):
//   warp 0     producer: 1-D bulk copies of the packed weight tiles (8 x 1 KB per 256-input
//              chunk) and of the chunk's int8 activation block into a shared-memory ring;
//   warp 1     MMA issuer (one thread): tcgen05.mma.kind::i8 with the A operand (weights, u8) in
//              TENSOR MEMORY and the B operand (activations, s8) in shared memory, K-major in the 64-byte
//              swizzle; accumulators in tensor memory, two sets where there is room, so that the MMAs of the
//              next unit run while the previous one is drained;
//   8 unpack warps: a thread owns one weight row (= one TMEM lane) of one row set (with one row set, two warps per
//              lane quarter take the chunks in turn).  It loads the row's 64
//              packed bytes of the chunk, isolates field r of every byte with a shift and an AND (values 0, 1, 2 =
//              ternary + 1) and writes the four residue planes with tcgen05.st straight into tensor memory:
//              the unpacked weights never pass through shared memory, whose bandwidth the B operand and the ring need;
//   4 RS epilogue warps: tcgen05.ld of a finished accumulator set, - sum_k q (the +1 offset), scales, store.
// With few output tiles the k range of a tile is cut over the CTAs of a thread-block cluster; their int32
// partial sums reach the cluster's first CTA through distributed shared memory, and that CTA alone stores.
// Every launch carries the programmatic-dependent-launch attribute: the producer requests the first weight
// tiles (which no kernel writes) before it waits for the kernel in front.
// A 2-bit field at position r of a byte multiplies the activations k = r (mod 4), hence the
// activations are stored residue-split: B_r[m, k'] = q[m, 4k' + r]; the four residue products of a
// chunk accumulate into the same accumulator.
#include <cstdint>
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "bt_common.cuh"
#include "bt_model.cuh"
#include "bt_ptx.cuh"

namespace bt {

namespace {

constexpr int kRows = 128;               // weight rows per MMA = UMMA M = TMEM lanes
constexpr int kSetBytes = 8 * kTileBytes;  // packed weights of 128 rows of a chunk: 8 row tiles x 1 KB
constexpr int kAChunkCols = 64;          // TMEM columns of one unpacked 128-row chunk: 4 residues x 64 bytes / 4
constexpr int kEpiBf16Accum = 100;       // the last of several bases with a bf16 output: bf16(acc_in + (acc * s_w) * s_x[m])
constexpr unsigned kErrTcTimeout = 0x54434d4du;  // 'TCMM'

// A tile is RS x 128 weight rows x NT tokens: the RS row sets share every activation block, which is what a CTA
// pulls most of through L2 (NT x 256 bytes per chunk against RS x 8 KB of packed weights).
// Warps: producer, MMA issuer, 8 unpack warps, 4 RS epilogue warps.  With two row sets two idle warps follow the MMA
// issuer, so that the roles fall on whole warpgroups (4 warps) and can trade registers (setmaxnreg).
__host__ __device__ constexpr int tc_lead_warps(int rs) { return rs == 2 ? 4 : 2; }
__host__ __device__ constexpr int tc_threads(int rs) { return (tc_lead_warps(rs) + 8 + 4 * rs) * 32; }
// Register split of the 128-token, two-row-set kernel: the epilogue warps hold a whole accumulator row (128 values) so
// that the single accumulator set is free again after four tensor-memory loads instead of after the stores.
constexpr int kRegsLead = 40, kRegsUnpack = 64, kRegsEpilogue = 152;
__host__ __device__ constexpr bool tc_reg_split(int nt, int rs, int s, bool pair) { return pair || (nt == 128 && rs == 2 && s == 1); }
__host__ __device__ constexpr int tc_abufs(int rs) { return rs == 1 ? 4 : 2; }           // unpacked-A buffers in tensor memory
__host__ __device__ constexpr int tc_acc_sets(int nt, int rs) { return (2 * rs * nt + tc_abufs(rs) * rs * kAChunkCols <= 512) ? 2 : 1; }
__host__ __device__ constexpr int tc_stages(int nt, int rs, int s) {
    // ring depth that fits 227 KB next to the partial-sum buffer of a k split
    const int stage = rs * kSetBytes + 4 * nt * 64, part = s > 1 ? rs * kRows * nt * 4 : 0;
    const int n = (225 * 1024 - part) / stage;
    return n > 5 ? 5 : n;
}

// A CTA pair's tile: 256 rows x 256 tokens, an MMA of 256 x 256 x 32 over both SMs.  Each CTA unpacks 128 rows and pulls in the
// activations of 128 of the tokens, which both tensor cores read: per product 160 bytes of a k step against the 192 of a single
// CTA's 256 x 128 tile, and half the unpacked weights and half the MMAs, whose issue and whose contention with the stores
// to tensor memory bound that tile (97 clocks of an MMA of 64).  A chunk of 256 inputs takes 1 400 to 1 900 clocks here, 1 032 of
// them MMAs; without its copies, or without its stores to tensor memory, or without the stores of the results it would be 5 to
// 20 % less (builds that are not in the tree): no single one bounds it.  Between two tiles the MMAs stop for 3 000 clocks, until
// the accumulators are in registers.
// Per launch, single CTAs -> pairs (us, f32 outputs): 2048 x 14336 -> 4096 129.2 -> 108.3, 4096 tokens 248 -> 202; 2048 x 4096 ->
// 4096 43.2 -> 40.0, -> 6144 60.6 -> 56.0; 2048 x 5632 -> 2048 31.8 -> 29.6; 2048 x 2048 -> 11264 57.6 -> 57.2.
constexpr int kPairTokens = 256;
constexpr int kPairChunks = 8;  // chunks of 256 inputs from which on pairs pay (see launch_product)

// Instruction descriptor for kind::i8: D = s32, A = u8, B = s8, both K-major, M x N tile.
__device__ __forceinline__ uint32_t instr_desc_i8(int m, int n) {
    uint32_t d = 0;
    d |= 2u << 4;                    // accumulator format: s32
    d |= 0u << 7;                    // A format: unsigned 8-bit
    d |= 1u << 10;                   // B format: signed 8-bit
    d |= (uint32_t)(n >> 3) << 17;   // N / 8
    d |= (uint32_t)(m >> 4) << 24;   // M / 16
    return d;
}

struct TcArgs {
    const uint8_t* tiles;      // one basis, tiled layout [row_tile][k_tile][1024]
    int64_t row_tiles, k_tiles, n_out;
    const int8_t* qtc;         // activations: [token_block][k_tile][4 residues][NT tokens][64], swizzled (gemm_tc_act_offset)
    const int32_t* qsum;       // [m]
    const float* sx;           // [m]
    const float* sw_tiles;     // [row_tiles][2]
    int m;                     // tokens
    void* out;                 // [m, out_stride]
    int64_t out_stride;
    int epilogue;              // EPI_I32 / EPI_F32 / EPI_F32_ACCUM / EPI_BF16 / kEpiBf16Accum
    const float* acc_in;       // what the accumulating epilogues add to: [m, out_stride] f32
    int bases;                 // up to 64 tokens: bases in this launch, one behind the other
    int64_t basis_bytes;       // from one basis' weights to the next
    float* sum;                // several bases and a bf16 output: [m, out_stride] f32, the bases so far
    unsigned int* err;
};

// NT: tokens per tile (64 / 128).  RS: 128-row sets per tile (1 / 2).  S: CTAs of a cluster that share a tile
// along k (1: no cluster work at all).
// PAIR: the cluster is a CTA pair that works on one tile of 256 rows x 256 tokens (see kPairTokens).
// SEVERAL: a.bases bases in this launch, one behind the other.  An instantiation of its own: with both epilogues in one kernel a
// product of a single basis had 88 to 128 registers a thread instead of 83 to 108, and the quantiser in front of it no longer
// fitted beside its CTA, which starts under it (64 tokens of the 8B shapes with their quantisers, us a step in runs of two kinds,
// by where the process' memory lies: 2 167 and 2 264, now 2 118 and 2 198).
template <int NT, int RS, int S, bool PAIR, bool SEVERAL>
__global__ void __launch_bounds__(tc_threads(PAIR ? 2 : RS), 1) gemm_tc_kernel(TcArgs a) {
    static_assert(S == 1 || (NT == 64 && (S == 2 || S == 4 || S == 8)), "k split: 64 tokens, 2 / 4 / 8 CTAs");
    static_assert(!PAIR || (NT == 128 && RS == 1 && S == 1), "a CTA of a pair: 128 rows and the activations of 128 tokens");
    static_assert(!SEVERAL || NT == 64, "larger products fill the GPU basis by basis");
    // Eight unpack warps.  RS = 2: one per (row set, TMEM lane quarter).  RS = 1: two per lane quarter, which take
    // the chunks in turn (two independent chains of load - unpack - store, four A buffers).
    constexpr int kUnpackWarps = 8, kEpiWarps = PAIR ? 8 : 4 * RS, kUnpackWarp0 = tc_lead_warps(PAIR ? 2 : RS), kEpiWarp0 = kUnpackWarp0 + kUnpackWarps;
    constexpr bool kRegSplit = tc_reg_split(NT, RS, S, PAIR);
    constexpr int kABufs = tc_abufs(RS);
    constexpr int kReaders = RS == 1 ? 4 : 8;            // unpack warps that read one stage's weights and fill one A buffer
    constexpr int kStages = tc_stages(NT, RS, S);
    constexpr int kAccSets = PAIR ? 1 : tc_acc_sets(NT, RS);
    constexpr int kRawBytes = RS * kSetBytes;
    constexpr int kBBytes = 4 * NT * 64;                 // activation block of a chunk (4 residues)
    constexpr int kStageBytes = kRawBytes + kBBytes;
    constexpr int kPartBytes = S > 1 ? RS * kRows * NT * 4 : 0;  // this CTA's partial sums of a tile, read by the whole cluster
    constexpr uint32_t kAccCols = PAIR ? kPairTokens : kAccSets * RS * NT;
    constexpr int kTokSets = PAIR ? 2 : 1;               // token halves of the tile, drained by different warps
    constexpr uint32_t kTmemCols = (kAccCols + kABufs * RS * kAChunkCols) <= 256 ? 256 : 512;
    static_assert(kAccCols + kABufs * RS * kAChunkCols <= 512, "tensor memory");
    static_assert(kStages >= 3, "ring");
    static_assert(RS == 2 || kStages % 2 == 0 || kStages > kABufs, "a set of unpack warps must not ask for a stage whose chunk before has not landed");
    extern __shared__ __align__(1024) uint8_t smem[];  // (the swizzle of the activation blocks goes by address bits 7 and 8)
    uint8_t* stage_base = smem;                                           // kStages x (raw | B)
    int32_t* pbuf = reinterpret_cast<int32_t*>(stage_base + (size_t)kStages * kStageBytes);  // [RS][NT / 4][128 rows][4]
    uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(pbuf) + kPartBytes);
    uint64_t* empty = full + kStages;     // a stage is free again: the MMAs that read its B block are done (1 arrival)
                                          // and the unpack warps that take the chunk have read its weights
    uint64_t* a_full = empty + kStages;   // unpacked chunk in tensor memory (one arrival per unpack warp)
    uint64_t* a_empty = a_full + kABufs;  // the MMAs that read it are done
    uint64_t* acc_full = a_empty + kABufs;
    uint64_t* acc_empty = acc_full + 2;   // one arrival per epilogue warp
    uint64_t* red_full = acc_empty + 2;   // every CTA of the cluster has parked its partial sums of the tile
    uint64_t* red_free = red_full + 1;    // every CTA of the cluster has read this CTA's partial sums
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(red_free + 1);
    int* tok_qsum = reinterpret_cast<int*>(tmem_slot + 2);          // [2][kTokSets][NT] per-token sum of q and scale of the tile being drained
    float* tok_sx = reinterpret_cast<float*>(tok_qsum + 2 * kTokSets * NT);  // (two copies: the row sets' warps may be one tile apart)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_tiles = (int)a.k_tiles;
    constexpr int kTileSets = PAIR ? 2 : RS, kTileTokens = PAIR ? kPairTokens : NT, kCtas = PAIR ? 2 : S;
    const int row_sets = (int)((a.row_tiles + 8 * kTileSets - 1) / (8 * kTileSets));   // tiles along the rows
    const int tok_blocks = (a.m + kTileTokens - 1) / kTileTokens;
    const int rank = kCtas > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int cid = blockIdx.x / kCtas, n_clusters = gridDim.x / kCtas;
    const int cps = (k_tiles + S - 1) / S;                 // chunks per split (the host makes every split non-empty)
    const int kt0 = PAIR ? 0 : rank * cps, kt1 = min(k_tiles, kt0 + cps);
    const int bases = SEVERAL ? a.bases : 1;               // a tile's bases are worked through like tiles of their own
    const int n_tiles = row_sets * tok_blocks;             // this CTA works on the tiles cid, cid + n_clusters, ...
    // this CTA's row tiles of a tile begin at row_tile0(rs): rts(rs) of them exist (none, where the matrix ends in the first half)
    auto row_tile0 = [&](int rs) -> int64_t { return (int64_t)rs * (8 * kTileSets) + (PAIR ? 8 * rank : 0); };
    auto row_tiles_of = [&](int rs) -> int { return max(0, min(8 * RS, (int)(a.row_tiles - row_tile0(rs)))); };

    if (warp == 0) {  // the barriers side by side, a lane each (the set-up is on the path of every launch)
        if (lane < kStages) { ptx::mbar_init(&full[lane], 1); ptx::mbar_init(&empty[lane], 1 + kReaders); }
        // (of a pair, rank 0's a_full and acc_empty count the warps of both CTAs)
        if (lane >= 8 && lane < 8 + kABufs) { ptx::mbar_init(&a_full[lane - 8], kReaders * (PAIR ? 2 : 1)); ptx::mbar_init(&a_empty[lane - 8], 1); }
        if (lane >= 16 && lane < 18) { ptx::mbar_init(&acc_full[lane - 16], 1); ptx::mbar_init(&acc_empty[lane - 16], kEpiWarps * (PAIR ? 2 : 1)); }
        if (lane == 24) ptx::mbar_init(red_full, kEpiWarps * S);
        if (lane == 25) ptx::mbar_init(red_free, kEpiWarps * S);
        ptx::mbar_fence_init();
    }
    if (warp == 1) {  // one warp allocates (and later frees) the tensor memory
        if constexpr (PAIR) { ptx::tmem_alloc_pair(tmem_slot, kTmemCols); ptx::tmem_relinquish_pair(); }
        else { ptx::tmem_alloc(tmem_slot, kTmemCols); ptx::tmem_relinquish(); }
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    // The peers' barriers must exist before anybody arrives on them.  Only the epilogue warps ever touch a peer, so
    // everybody reports here and only they wait (at the top of their role): the cluster's start-up skew stays off
    // the path of the first copies and MMAs.  (Of a pair every warp waits, the producer after its first requests: the
    // unpack warps and the commits arrive on the peer's barriers too, and the closing cluster barrier takes everybody.)
    if (S > 1 || PAIR) ptx::cluster_arrive();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t a_col0 = kAccCols;  // the unpacked-A buffers follow the accumulators: [buffer][row set][64]

    // With the register split every warpgroup states its share at the top of its branch (the host has checked that the
    // shares fit the register file the launch gives the CTA).
    bool ok = true;
    if (warp < kUnpackWarp0) {
    if constexpr (kRegSplit) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsLead));
    if (warp == 0) {
        // ---------------- producer (whole warp: lane r8 requests row tile r8 of a chunk, so that the small copies are
        //                  issued side by side; lane 0 also registers the byte count and requests the activation block) ----
        {
            // The weights do not depend on earlier kernels: the first stages' weight tiles are requested before the
            // dependency wait, their activation blocks (written by the quantiser just before) after it.
            auto issue = [&](int tile, int basis, int kt, int slot, bool raw_part, bool b_part) {
                const int rs = tile % row_sets, tb = tile / row_sets;
                uint8_t* st = stage_base + (size_t)slot * kStageBytes;
                const int rts = row_tiles_of(rs);
                if (raw_part) {
                    if (lane == 0) ptx::mbar_arrive_expect_tx(&full[slot], (uint32_t)(rts * kTileBytes + kBBytes));
                    if (lane < rts)
                        ptx::bulk_g2s(st + lane * kTileBytes, a.tiles + basis * a.basis_bytes + ((row_tile0(rs) + lane) * k_tiles + kt) * kTileBytes, kTileBytes,
                                      &full[slot]);
                }
                // (a pair's second half may lie behind the last token block: it reads that block again, nothing of it is stored)
                const int blk = PAIR ? min(2 * tb + rank, (a.m + NT - 1) / NT - 1) : tb;
                if (b_part && lane == 0) ptx::bulk_g2s(st + kRawBytes, a.qtc + ((int64_t)blk * k_tiles + kt) * kBBytes, kBBytes, &full[slot]);
            };
            int g = 0;
            for (int tile = cid; tile < n_tiles && g < kStages; tile += n_clusters)
                for (int basis = 0; basis < bases; ++basis)
                    for (int kt = kt0; kt < kt1 && g < kStages; ++kt, ++g) issue(tile, basis, kt, g, true, false);
            if constexpr (PAIR) { __syncwarp(); ptx::cluster_wait(); }
            ptx::pdl_wait();
            g = 0;
            for (int tile = cid; tile < n_tiles; tile += n_clusters)
            for (int basis = 0; basis < bases; ++basis) {
                for (int kt = kt0; kt < kt1; ++kt, ++g) {
                    const int slot = g % kStages, use = g / kStages;
                    if (use == 0) { issue(tile, basis, kt, slot, false, true); continue; }
                    ok &= ptx::mbar_wait_bounded(&empty[slot], (uint32_t)((use - 1) & 1));
                    issue(tile, basis, kt, slot, true, true);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (of a pair: rank 0's) ----------------
        if constexpr (PAIR) ptx::cluster_wait();
        if (PAIR && rank != 0) {
            if (lane == 0) ptx::pdl_launch_dependents();  // (rank 0 issues the MMAs and says when the kernel behind may start)
        } else if (lane == 0) {
            ptx::pdl_wait();  // nothing to do before the first activation block exists; keeps the bounded waits short
            const uint32_t idesc = PAIR ? instr_desc_i8(2 * kRows, kPairTokens) : instr_desc_i8(kRows, NT);
            auto commit = [&](uint64_t* bar) {
                if constexpr (PAIR) ptx::umma_commit_pair(bar);
                else ptx::umma_commit(bar);
            };
            int g = 0, tl = 0;
            for (int tile = cid; tile < n_tiles; tile += n_clusters)
            for (int basis = 0; basis < bases; ++basis, ++tl) {
                const int sel = tl % kAccSets, acc_use = tl / kAccSets;
                if constexpr (PAIR) { if (acc_use > 0) ok &= ptx::mbar_spin_cluster(&acc_empty[sel], (uint32_t)((acc_use - 1) & 1)); }
                else if (acc_use > 0) ok &= ptx::mbar_wait_bounded(&acc_empty[sel], (uint32_t)((acc_use - 1) & 1));
                ptx::tc_fence_after();
                for (int kt = kt0; kt < kt1; ++kt, ++g) {
                    const int slot = g % kStages, u = g % kABufs;
                    // One wait per chunk: the unpack warps arrive on a_full after they have seen full[slot] complete, which
                    // covers the stage's activation block as well as its weights.  Every instruction between two MMAs
                    // of this thread costs tensor-pipe time (the queue behind it is short), hence the relaxed wait.
                    // (A pair's wait acquires at cluster scope: the peer's warps arrive too, for weights in its tensor memory and activations
                    // in its shared memory.  The acquire costs nothing here, relaxed -> acquired us: 4096 x 14336 -> 4096 259.2 -> 255.9,
                    // 2048 x 4096 -> 6144 60.8 -> 60.2; a relaxed wait with a cluster fence behind it 365.7 and 82.4.)
                    if constexpr (PAIR) ok &= ptx::mbar_spin_cluster(&a_full[u], (uint32_t)((g / kABufs) & 1));
                    else ok &= ptx::mbar_spin_relaxed(&a_full[u], (uint32_t)((g / kABufs) & 1));  // weights unpacked into tensor memory
                    ptx::tc_fence_after();
                    const uint32_t b_addr = ptx::smem_u32(stage_base + (size_t)slot * kStageBytes + kRawBytes);
#pragma unroll
                    for (int h = 0; h < RS; ++h) {
                        const uint32_t d_tmem = tmem_base + (uint32_t)(sel * RS + h) * NT;
                        const uint32_t a_tmem = tmem_base + a_col0 + (uint32_t)(u * RS + h) * kAChunkCols;
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
#pragma unroll
                            for (int ks = 0; ks < 2; ++ks) {  // 64 k' per residue = 2 x K32 = 2 x 8 TMEM columns
                                const uint64_t bd = ptx::smem_desc_sw64(b_addr + r * (NT * 64) + ks * 32, 512);
                                const uint32_t add = (kt > kt0 || r > 0 || ks > 0) ? 1u : 0u;
                                if constexpr (PAIR) ptx::umma_i8_ts_pair(d_tmem, a_tmem + r * 16 + ks * 8, bd, idesc, add);
                                else ptx::umma_i8_ts(d_tmem, a_tmem + r * 16 + ks * 8, bd, idesc, add);
                            }
                        }
                    }
                    commit(&a_empty[u]);   // unpacked buffer reusable once these MMAs are done
                    commit(&empty[slot]);  // and the stage's activation block
                }
                commit(&acc_full[sel]);
            }
            // every MMA of this CTA is issued: the kernel behind may start (it waits for this one's results itself)
            ptx::pdl_launch_dependents();
        }
    } else {
        if constexpr (PAIR) ptx::cluster_wait();  // (the idle warps of the leading warpgroup)
    }
    } else if (warp < kEpiWarp0) {
        if constexpr (kRegSplit) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsUnpack));
        // ---------------- unpack warps: a thread owns one weight row (= one TMEM lane) of one row set ----
        const int sub = warp & 3;                      // the TMEM lanes 32 sub .. 32 sub + 31 belong to this warp
        const int set = (warp - kUnpackWarp0) >> 2;               // RS = 2: row set of the tile; RS = 1: which chunks (even / odd)
        const int h = RS == 2 ? set : 0;
        const int row = sub * 32 + lane;               // row inside the set
        // the row: row tile r8 = row/16, half = (row%16)/8, g = row%8; its 64 packed bytes of a chunk are the four
        // 16-byte pieces t = 0..3 at ((half*32 + g*4 + t) * 16) of the row tile
        const int r8 = h * 8 + (row >> 4), half = (row >> 3) & 1, g8 = row & 7;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(sub * 32) << 16) + a_col0 + (uint32_t)h * kAChunkCols;
        if constexpr (PAIR) ptx::cluster_wait();
        ptx::pdl_wait();
        int g = 0;
        int pending = -1;  // A buffer whose stores are issued but not yet published
        // The stores of a chunk are published (wait, fence, arrive) only after the next chunk's weights have been
        // loaded from shared memory, if those have landed already: the store latency hides behind the loads.
        auto publish = [&]() {
            if (pending < 0) return;
            ptx::tmem_st_wait();
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (PAIR) ptx::mbar_arrive_remote(ptx::map_to_rank(&a_full[pending], 0));
                else ptx::mbar_arrive(&a_full[pending]);
            }
            pending = -1;
        };
        for (int tile = cid; tile < n_tiles; tile += n_clusters)
        for (int basis = 0; basis < bases; ++basis) {
            const int rs = tile % row_sets;
            const int rts = row_tiles_of(rs);
            for (int kt = kt0; kt < kt1; ++kt, ++g) {
                if (RS == 1 && (g & 1) != set) continue;
                const int slot = g % kStages, u = g % kABufs, a_use = g / kABufs;
                const uint32_t full_parity = (uint32_t)((g / kStages) & 1), buffer_parity = (uint32_t)((a_use - 1) & 1);
                // RS = 1: the buffer before the weights.  The chunk that lay in this stage before belongs to the other set (kStages is odd),
                // and while its copies were still on their way the parity asked for below would be granted for the phase before
                // them.  The buffer's last product, kABufs chunks back, came after that chunk's.  (A ring of four stages, in which a set
                // meets the same stages again and again, takes the same time with single CTAs, but 2048 x 14336 -> 4096 142 us with
                // pairs, and 133 like this.)
                if (RS == 1 && a_use > 0 && !__all_sync(0xffffffffu, ptx::mbar_test_wait(&a_empty[u], buffer_parity))) {
                    publish();
                    ok &= ptx::mbar_wait_bounded(&a_empty[u], buffer_parity);
                }
                if (!__all_sync(0xffffffffu, ptx::mbar_test_wait(&full[slot], full_parity))) {  // (one answer for the whole warp)
                    publish();  // the next weights are not here yet: do not hold the finished buffer back
                    ok &= ptx::mbar_wait_bounded(&full[slot], full_parity);
                }
                const uint8_t* raw = stage_base + (size_t)slot * kStageBytes + r8 * kTileBytes + half * 512 + g8 * 64;
                uint4 w[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    w[t] = make_uint4(0x55555555u, 0x55555555u, 0x55555555u, 0x55555555u);  // weight 0 (rows beyond the matrix)
                    if (r8 < rts) w[t] = *reinterpret_cast<const uint4*>(raw + t * 16);
                }
                publish();
                if (RS == 2 && a_use > 0) ok &= ptx::mbar_wait_bounded(&a_empty[u], buffer_parity);
                ptx::tc_fence_after();
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    // residue r: piece t holds the inputs 64 t .. 64 t + 63, i.e. k' = 16 t .. 16 t + 15 = columns 4 t .. 4 t + 3
                    uint32_t v[16];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        v[4 * t + 0] = (w[t].x >> (2 * r)) & 0x03030303u;
                        v[4 * t + 1] = (w[t].y >> (2 * r)) & 0x03030303u;
                        v[4 * t + 2] = (w[t].z >> (2 * r)) & 0x03030303u;
                        v[4 * t + 3] = (w[t].w >> (2 * r)) & 0x03030303u;
                    }
                    ptx::tmem_st16(lane_addr + (uint32_t)(u * RS) * kAChunkCols + r * 16, v);
                }
                pending = u;
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&empty[slot]);  // this warp holds the stage's weights in registers
            }
        }
        publish();
    } else {
        if constexpr (kRegSplit) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
        // ---------------- epilogue warps (4 per row set, TMEM lanes by warp % 4) ----------------
        const int sub = warp & 3;
        const int h = (warp - kEpiWarp0) >> 2;  // row set of the tile; of a pair: token half
        const int lrow = sub * 32 + lane;       // row inside the set
        int32_t* pb = pbuf + (size_t)h * (kRows * NT);
        if (S > 1 || PAIR) ptx::cluster_wait();
        ptx::pdl_wait();  // the output (and what EPI_F32_ACCUM adds to) belongs to earlier kernels until here
        // The old value of an accumulated output is fetched apart from its update, so that a thread's loads are all
        // in flight before the first store (a store followed by a load of the same array would serialise them);
        // the per-token terms come through the read-only path for the same reason.
        // The epilogue kind is a compile-time constant of everything below (one copy of the role per kind, chosen once):
        // the unrolled store sequences are long, and a kind switch inside every element made them four times as long -
        // code that is fetched once per tile and does not stay in the instruction cache.
        // Several bases are added up in basis order in f32 rows (the output, or aside before a bf16 output); the thread that
        // adds a basis is the one that stored the one before.
        auto epilogue_role = [&](auto kind) {
        constexpr int EPI = decltype(kind)::value;
        constexpr bool accum = SEVERAL || EPI == EPI_F32_ACCUM || EPI == kEpiBf16Accum;
        int basis = 0;
        auto load_old = [&](int token, int64_t row) -> float {
            if constexpr (SEVERAL) {
                const int64_t o = (int64_t)token * a.out_stride + row;
                if (basis == 0 || token >= a.m || row >= a.n_out) return 0.0f;
                return EPI == EPI_BF16 ? a.sum[o] : reinterpret_cast<const float*>(a.out)[o];
            } else {
                return (accum && token < a.m && row < a.n_out) ? a.acc_in[(int64_t)token * a.out_stride + row] : 0.0f;
            }
        };
        // i = token inside the tile; tq / ts = the tile's staged per-token terms
        // tqi / tsi: the token's sum of q and scale (read from shared memory by the caller, ahead of its stores)
        // (tok0: the first token of those that this warp drains)
        auto store_v = [&](int tqi, float tsi, int tok0, int i, int n_tok, int64_t row, float sw, uint32_t acc, float old) {
            if (i < n_tok && row < a.n_out) {
                const int accv = (int)acc - tqi;
                const int64_t o = (int64_t)(tok0 + i) * a.out_stride + row;
                if constexpr (EPI == EPI_I32) {
                    reinterpret_cast<int32_t*>(a.out)[o] = accv;
                } else {
                    const float y = __fmul_rn(__fmul_rn((float)accv, sw), tsi);
                    if constexpr (SEVERAL) {
                        const float v = basis == 0 ? y : __fadd_rn(old, y);
                        if (EPI == EPI_F32) reinterpret_cast<float*>(a.out)[o] = v;
                        else if (basis + 1 < a.bases) a.sum[o] = v;
                        else reinterpret_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(v);
                    } else if constexpr (EPI == EPI_F32) reinterpret_cast<float*>(a.out)[o] = y;
                    else if constexpr (EPI == EPI_F32_ACCUM) reinterpret_cast<float*>(a.out)[o] = __fadd_rn(old, y);
                    else if constexpr (EPI == kEpiBf16Accum) reinterpret_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(__fadd_rn(old, y));
                    else reinterpret_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16_rn(y);
                }
            }
        };
        auto store = [&](const int* tq, const float* ts, int tok0, int i, int n_tok, int64_t row, float sw, uint32_t acc, float old) {
            store_v(tq[i], ts[i], tok0, i, n_tok, row, sw, acc, old);
        };
        // EPI_SWIGLU: rows 0-7 of a row tile are gate rows, rows 8-15 the matching up rows, eight lanes further on.  Of `half` + half
        // tokens in a lane's registers the gate lane finishes the first half and the up lane the second, so that both compute:
        // each sends what the other needs.  f32 as in the quantiser that did this before (silu(g) * u, layers/swiglu.rs:31-33).
        auto swiglu = [&](uint32_t mine, uint32_t other, int tqi, float tsi, float sw_gate, float sw_up, bool up) -> float {
            const float g = __fmul_rn(__fmul_rn((float)((int)(up ? other : mine) - tqi), sw_gate), tsi);
            const float u = __fmul_rn(__fmul_rn((float)((int)(up ? mine : other) - tqi), sw_up), tsi);
            return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u);
        };
        // a set of accumulator columns has been read: the MMA issuer may write it again
        auto free_set = [&](int sel) {
            if constexpr (PAIR) ptx::mbar_arrive_remote(ptx::map_to_rank(&acc_empty[sel], 0));
            else ptx::mbar_arrive(&acc_empty[sel]);
        };
        int tl = 0;
        for (int tile = cid; tile < n_tiles; tile += n_clusters)
        for (basis = 0; basis < bases; ++basis, ++tl) {
            const int rs = tile % row_sets, tb = tile / row_sets;
            const int sel = tl % kAccSets;
            // the tile's per-token terms, once per row set's four warps into shared memory (named barrier 1 + h)
            const int tok0 = PAIR ? tb * kPairTokens + h * NT : tb * NT;
            const int tset = ((tl & 1) * kTokSets + (PAIR ? h : 0)) * NT;
            {
                int* tq = tok_qsum + tset;
                float* ts = tok_sx + tset;
                if (h == 0 || RS == 1) {
                    for (int i = lrow; i < NT; i += kRows) {
                        const int token = tok0 + i;
                        tq[i] = token < a.m ? __ldg(a.qsum + token) : 0;
                        ts[i] = (token < a.m && EPI != EPI_I32) ? __ldg(a.sx + token) : 0.0f;
                    }
                }
                ptx::named_bar_sync(1, kEpiWarps * 32);  // all epilogue warps: written before read, read before the tile after next overwrites
            }
            ok &= ptx::mbar_wait_bounded(&acc_full[sel], (uint32_t)((tl / kAccSets) & 1));
            ptx::tc_fence_after();
            const int* tq = tok_qsum + tset;
            const float* ts = tok_sx + tset;
            const int64_t row = PAIR ? ((int64_t)rs * 2 + rank) * kRows + lrow : ((int64_t)rs * RS + h) * kRows + lrow;
            const int64_t rt = row >> 4;
            float sw = 0.f;
            if (EPI != EPI_I32 && rt < a.row_tiles) sw = __ldg(a.sw_tiles + 2 * (basis * a.row_tiles + rt) + ((row >> 3) & 1));
            const uint32_t acc_addr = tmem_base + ((uint32_t)(sub * 32) << 16) + (uint32_t)(sel * RS + h) * NT;
            const int n_tok = min(NT, a.m - tok0);  // tokens of these that exist
            bool drained = false;
            if constexpr (kRegSplit && EPI != EPI_I32) {
                // Whole tiles: this thread's whole accumulator row goes to registers and the set is handed back to the MMA
                // issuer before the first store, so that the next tile's MMAs run under this tile's stores (the loop
                // below holds them back: 2048 x 4096 -> 28672 with a bf16 output 297 us there, 229 here).  The store
                // code is kept short (one epilogue kind per loop, no per-element bounds): it is unrolled 128 times and is
                // fetched once per tile.
                // (one decision per warp: the tensor-memory loads are warp-wide instructions)
                if (n_tok == NT && __all_sync(0xffffffffu, row < a.n_out)) {
                    drained = true;
                    uint32_t d[NT];
#pragma unroll
                    for (int c0 = 0; c0 < NT; c0 += 32) ptx::tmem_ld32(acc_addr + c0, reinterpret_cast<uint32_t(&)[32]>(d[c0]));
                    ptx::tmem_ld_wait();
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) free_set(sel);
                    using Out = std::conditional_t<EPI == EPI_BF16 || EPI == kEpiBf16Accum, __nv_bfloat16, float>;
                    const int64_t stride = a.out_stride, at = (int64_t)tok0 * stride + row;
                    if constexpr (EPI == EPI_SWIGLU) {
                        const bool up = lane & 8;
                        const float sw_other = __shfl_xor_sync(0xffffffffu, sw, 8), sw_gate = up ? sw_other : sw, sw_up = up ? sw : sw_other;
                        const int *tqh = tq + (up ? NT / 2 : 0);
                        const float *tsh = ts + (up ? NT / 2 : 0);
                        float* po = reinterpret_cast<float*>(a.out) + (int64_t)(tok0 + (up ? NT / 2 : 0)) * stride + (row >> 4) * 8 + (row & 7);
#pragma unroll
                        for (int i = 0; i < NT / 2; ++i) {
                            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? d[i] : d[NT / 2 + i], 8);
                            po[i * stride] = swiglu(up ? d[NT / 2 + i] : d[i], got, tqh[i], tsh[i], sw_gate, sw_up, up);
                        }
                    } else {
                    Out* po = reinterpret_cast<Out*>(a.out) + at;
                    auto put = [&](int i, float y) {
                        if constexpr (std::is_same_v<Out, float>) po[i * stride] = y;
                        else po[i * stride] = __float2bfloat16_rn(y);
                    };
                    if (accum) {
                        const float* pi = a.acc_in + at;
#pragma unroll
                        for (int c0 = 0; c0 < NT; c0 += 16) {
                            float old[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) old[j] = pi[(c0 + j) * stride];
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                put(c0 + j, __fadd_rn(old[j], __fmul_rn(__fmul_rn((float)((int)d[c0 + j] - tq[c0 + j]), sw), ts[c0 + j])));
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < NT; ++i) put(i, __fmul_rn(__fmul_rn((float)((int)d[i] - tq[i]), sw), ts[i]));
                    }
                    }
                }
            }
            if (drained) {
                // nothing left to do for this tile
            } else if constexpr (S == 1) {
                if constexpr (EPI == EPI_SWIGLU) {
                    const bool up = lane & 8;
                    const float sw_other = __shfl_xor_sync(0xffffffffu, sw, 8), sw_gate = up ? sw_other : sw, sw_up = up ? sw : sw_other;
                    const int64_t col = (row >> 4) * 8 + (row & 7);
#pragma unroll 1
                    for (int c0 = 0; c0 < NT; c0 += 32) {
                        uint32_t d[32];
                        ptx::tmem_ld32(acc_addr + c0, d);
                        ptx::tmem_ld_wait();
                        const int i0 = c0 + (up ? 16 : 0);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? d[j] : d[16 + j], 8);
                            if (i0 + j < n_tok && row < a.n_out)
                                reinterpret_cast<float*>(a.out)[(int64_t)(tok0 + i0 + j) * a.out_stride + col] = swiglu(up ? d[16 + j] : d[j], got, tq[i0 + j], ts[i0 + j], sw_gate, sw_up, up);
                        }
                        __syncwarp();
                    }
                } else if (accum) {
#pragma unroll 1
                    for (int c0 = 0; c0 < NT; c0 += 16) {
                        uint32_t d[16];
                        float old[16];
                        ptx::tmem_ld16(acc_addr + c0, d);
#pragma unroll
                        for (int j = 0; j < 16; ++j) old[j] = load_old(tok0 + c0 + j, row);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) store(tq, ts, tok0, c0 + j, n_tok, row, sw, d[j], old[j]);
                    }
                } else {
#pragma unroll 1
                    for (int c0 = 0; c0 < NT; c0 += 32) {
                        uint32_t d[32];
                        ptx::tmem_ld32(acc_addr + c0, d);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) store(tq, ts, tok0, c0 + j, n_tok, row, sw, d[j], 0.0f);
                    }
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) free_set(sel);
            } else {
                // Reduce-scatter over the cluster: every CTA parks its partial sums of the whole tile in its own
                // shared memory ([row set][token / 4][row][token % 4], 16 bytes per thread and step), then adds up and
                // stores the NT / S tokens that are its share, reading all S copies through distributed shared memory.
                if (tl > 0) ok &= ptx::mbar_wait_cluster_bounded(red_free, (uint32_t)((tl - 1) & 1));  // everybody has read the previous tile
#pragma unroll 1
                for (int c0 = 0; c0 < NT; c0 += 32) {
                    uint32_t d[32];
                    ptx::tmem_ld32(acc_addr + c0, d);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<uint4*>(pb + ((size_t)(c0 / 4 + q) * kRows + lrow) * 4) =
                            make_uint4(d[4 * q], d[4 * q + 1], d[4 * q + 2], d[4 * q + 3]);
                }
                ptx::tc_fence_before();
                ptx::fence_cluster();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive(&acc_empty[sel]);  // the accumulator set is free for a later tile
                    // (the fence above has published the parked sums: the arrivals need no release of their own)
#pragma unroll
                    for (int pr = 0; pr < S; ++pr) ptx::mbar_arrive_remote_relaxed(ptx::map_to_rank(red_full, (uint32_t)pr));
                }
                ok &= ptx::mbar_wait_cluster_bounded(red_full, (uint32_t)(tl & 1));  // all S copies are complete
                constexpr int kGroups = NT / 4 / S;  // groups of 4 tokens that this CTA finishes
                constexpr int kBatch = 8 / S;        // groups per round: 8 remote 16-byte loads in flight
#pragma unroll 1
                for (int q0 = 0; q0 < kGroups; q0 += kBatch) {
                    float old[kBatch][4];
                    uint4 part[kBatch][S];
#pragma unroll
                    for (int q = 0; q < kBatch; ++q)
#pragma unroll
                        for (int pr = 0; pr < S; ++pr)
                            part[q][pr] = ptx::ld_dsmem_v4(
                                ptx::map_to_rank(pb + ((size_t)(rank * kGroups + q0 + q) * kRows + lrow) * 4, (uint32_t)pr));
#pragma unroll
                    for (int q = 0; q < kBatch; ++q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) old[q][e] = load_old(tok0 + (rank * kGroups + q0 + q) * 4 + e, row);
                    // the per-token terms too: a shared-memory load between two global stores would wait for the store
                    int tqv[kBatch][4];
                    float tsv[kBatch][4];
#pragma unroll
                    for (int q = 0; q < kBatch; ++q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            tqv[q][e] = tq[(rank * kGroups + q0 + q) * 4 + e];
                            tsv[q][e] = ts[(rank * kGroups + q0 + q) * 4 + e];
                        }
#pragma unroll
                    for (int q = 0; q < kBatch; ++q) {
                        uint4 s = part[q][0];
#pragma unroll
                        for (int pr = 1; pr < S; ++pr) {
                            s.x += part[q][pr].x; s.y += part[q][pr].y; s.z += part[q][pr].z; s.w += part[q][pr].w;
                        }
                        const int i = (rank * kGroups + q0 + q) * 4;
                        store_v(tqv[q][0], tsv[q][0], tok0, i, n_tok, row, sw, s.x, old[q][0]);
                        store_v(tqv[q][1], tsv[q][1], tok0, i + 1, n_tok, row, sw, s.y, old[q][1]);
                        store_v(tqv[q][2], tsv[q][2], tok0, i + 2, n_tok, row, sw, s.z, old[q][2]);
                        store_v(tqv[q][3], tsv[q][3], tok0, i + 3, n_tok, row, sw, s.w, old[q][3]);
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    // the peers' sums have been read and used: nothing of this thread is left to order
#pragma unroll
                    for (int pr = 0; pr < S; ++pr) ptx::mbar_arrive_remote_relaxed(ptx::map_to_rank(red_free, (uint32_t)pr));
                }
            }
        }
        };
        if constexpr (SEVERAL) {
            if (a.epilogue == EPI_F32) epilogue_role(std::integral_constant<int, EPI_F32>{});
            else epilogue_role(std::integral_constant<int, EPI_BF16>{});
        } else {
            switch (a.epilogue) {
                case EPI_I32: epilogue_role(std::integral_constant<int, EPI_I32>{}); break;
                case EPI_F32: epilogue_role(std::integral_constant<int, EPI_F32>{}); break;
                case EPI_F32_ACCUM: epilogue_role(std::integral_constant<int, EPI_F32_ACCUM>{}); break;
                case kEpiBf16Accum: epilogue_role(std::integral_constant<int, kEpiBf16Accum>{}); break;
                case EPI_SWIGLU: if constexpr (NT == 128 && (RS == 2 || PAIR)) epilogue_role(std::integral_constant<int, EPI_SWIGLU>{}); break;
                default: epilogue_role(std::integral_constant<int, EPI_BF16>{}); break;
            }
        }
    }
    if (!ok) atomicExch(a.err, kErrTcTimeout);
    ptx::tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) {
        // nobody leaves while the peer may still arrive on its barriers or its MMAs touch this CTA's memory
        ptx::cluster_arrive();
        ptx::cluster_wait();
        if (warp == 1) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    } else if (warp == 1) {
        ptx::tmem_dealloc(tmem_base, kTmemCols);
    }
    if (S > 1) {
        // Nobody leaves while a peer may still read its shared memory or arrive on its barriers: the last of both is
        // the peers' arrival on red_free for this CTA's last tile (they read the parked sums before it, and arrived on
        // red_full before that).  One warp waits for it; the CTA lives as long as that warp.
        const int my_tiles = cid < n_tiles ? (n_tiles - cid + n_clusters - 1) / n_clusters * bases : 0;
        if (warp == 2 && my_tiles > 0 && !ptx::mbar_wait_cluster_bounded(red_free, (uint32_t)((my_tiles - 1) & 1)))
            atomicExch(a.err, kErrTcTimeout);
    }
}

// One kernel variant (token tile NT, RS row sets per tile, S CTAs per cluster): its shared memory and how many
// clusters fit on the GPU at once (a cluster lives inside one GPC, so this is not SMs / S), asked of the runtime once.
struct TcVariant {
    size_t smem = 0;
    int max_clusters = 0;
    cudaError_t status = cudaErrorNotReady;
};

template <int NT, int RS, int S, bool PAIR = false, bool SEVERAL = false>
const TcVariant& tc_variant(int sm_count) {
    static TcVariant v;              // cluster limit: once per process (every device of a process is the same GPU model)
    static PerDeviceOnce attributes;  // the kernel's shared-memory limit: once per device
    constexpr int kCtas = PAIR ? 2 : S, kThreads = tc_threads(PAIR ? 2 : RS);
    v.smem = (size_t)tc_stages(NT, RS, S) * (RS * kSetBytes + 4 * NT * 64) + (S > 1 ? RS * kRows * NT * 4 : 0) + 512 + (PAIR ? 32 : 16) * NT;
    auto* kernel = gemm_tc_kernel<NT, RS, S, PAIR, SEVERAL>;
    const size_t smem = v.smem;
    v.status = attributes.run([kernel, smem] {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess && tc_reg_split(NT, RS, S, PAIR)) {
            // the register shares the warpgroups ask for must fit what the launch gives the CTA, or the asking waits for ever
            cudaFuncAttributes fa;
            e = cudaFuncGetAttributes(&fa, kernel);
            const int have = fa.numRegs * kThreads;
            const int want = 128 * kRegsLead + 256 * kRegsUnpack + 256 * kRegsEpilogue;
            if (e == cudaSuccess && have < want) e = cudaErrorLaunchOutOfResources;
        }
        return e;
    });
    if (v.status != cudaSuccess) return v;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (v.max_clusters != 0) return v;
    if (kCtas == 1) { v.max_clusters = sm_count; return v; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count / kCtas * kCtas));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = v.smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)kCtas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
        (void)cudaGetLastError();
        n = -1;  // this cluster size cannot be used
    }
    v.max_clusters = n;
    return v;
}

template <int NT, int RS, int S, bool PAIR = false, bool SEVERAL = false>
cudaError_t launch_variant(TcArgs a, int sm_count, cudaStream_t stream) {
    const TcVariant& v = tc_variant<NT, RS, S, PAIR, SEVERAL>(sm_count);
    if (v.status != cudaSuccess) return v.status;
    constexpr int kCtas = PAIR ? 2 : S, kSets = PAIR ? 2 : RS, kTokens = PAIR ? kPairTokens : NT;
    const int n_tiles = (int)((a.row_tiles + 8 * kSets - 1) / (8 * kSets)) * ((a.m + kTokens - 1) / kTokens);
    const int n_clusters = v.max_clusters < n_tiles ? v.max_clusters : n_tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_clusters * kCtas));
    cfg.blockDim = dim3(tc_threads(kSets));
    cfg.dynamicSmemBytes = v.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)kCtas; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = kCtas > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_tc_kernel<NT, RS, S, PAIR, SEVERAL>, a);
}

// Chunk steps on the busiest CTA when a tile's k range is cut over `s` CTAs (one step charged for the exchange of
// partial sums); a huge number when the cut is not possible.
int64_t tc_split_cost(int s, int max_clusters, int n_tiles, int64_t k_tiles) {
    if (max_clusters < 1) return INT64_MAX;  // (-1: the cluster size is unusable)
    const int64_t cps = (k_tiles + s - 1) / s;
    if (s > 1 && (k_tiles < 2 * s || cps * (s - 1) >= k_tiles)) return INT64_MAX;  // a CTA would be left without chunks
    const int nc = max_clusters < n_tiles ? max_clusters : n_tiles;
    return (int64_t)((n_tiles + nc - 1) / nc) * (cps + (s > 1 ? 1 : 0));
}

// 64 tokens at most.  More 128-row tiles than SMs: 256-row tiles.  Fewer than half: cut k over a cluster so that
// one wave of CTAs covers the product.
template <bool SEVERAL>
cudaError_t launch_product_64(TcArgs a, int sm_count, cudaStream_t stream) {
    const int n_tiles = (int)((a.row_tiles + 7) / 8);  // tiles of 128 rows
    if (n_tiles > sm_count) return launch_variant<64, 2, 1, false, SEVERAL>(a, sm_count, stream);
    int best = 1;
    int64_t best_cost = tc_split_cost(1, sm_count, n_tiles, a.k_tiles);
    if (n_tiles * 2 <= sm_count) {
        const int64_t c2 = tc_split_cost(2, tc_variant<64, 1, 2, false, SEVERAL>(sm_count).max_clusters, n_tiles, a.k_tiles);
        const int64_t c4 = tc_split_cost(4, tc_variant<64, 1, 4, false, SEVERAL>(sm_count).max_clusters, n_tiles, a.k_tiles);
        const int64_t c8 = tc_split_cost(8, tc_variant<64, 1, 8, false, SEVERAL>(sm_count).max_clusters, n_tiles, a.k_tiles);
        if (c2 < best_cost) { best = 2; best_cost = c2; }
        if (c4 < best_cost) { best = 4; best_cost = c4; }
        if (c8 < best_cost) { best = 8; best_cost = c8; }
    }
    switch (best) {
        case 2: return launch_variant<64, 1, 2, false, SEVERAL>(a, sm_count, stream);
        case 4: return launch_variant<64, 1, 4, false, SEVERAL>(a, sm_count, stream);
        case 8: return launch_variant<64, 1, 8, false, SEVERAL>(a, sm_count, stream);
        default: return launch_variant<64, 1, 1, false, SEVERAL>(a, sm_count, stream);
    }
}

cudaError_t launch_product(TcArgs a, int nt, int sm_count, cudaStream_t stream) {
    if (nt == 64) return a.bases > 1 ? launch_product_64<true>(a, sm_count, stream) : launch_product_64<false>(a, sm_count, stream);
    const int n_tiles2 = (int)((a.row_tiles + 15) / 16) * ((a.m + nt - 1) / nt);  // tiles of 256 rows
    // Pairs where there are tiles for most SMs and no more rounds of them than of single CTAs' tiles, which are half as large
    // (257 x 4096 -> 28672 has one more: 59.7 -> 68.7 us).  More than 16384 rows of plain output stay with single CTAs: their
    // stores, 1 KB of a token at a time instead of 512 bytes, disturb the loads less (2048 x 4096 -> 28672 233 us and 240);
    // with SiLU * up, which stores half of that, pairs are ahead again (prefill of 2048 tokens, 8B: 3 242 us and 3 290).  Fewer than 2048
    // inputs stay with single CTAs too, because a pair's tile ends in 3 000 clocks without MMAs and is twice as large: over 200 to
    // 4096 tokens and 2048 to 16384 rows pairs take 1.08 to 1.24 of their time for 256 inputs, 1.02 to 1.16 for 768, 0.96 to 1.05 for
    // 1280 and for 1536, 0.95 to 1.02 for 2048 (but 1354 x 2048 -> 10722: 1.08).
    const TcVariant& pair = tc_variant<128, 1, 1, true>(sm_count);
    const int n_pairs = (int)((a.row_tiles + 15) / 16) * ((a.m + kPairTokens - 1) / kPairTokens);
    // 256-row tiles halve the activation traffic per weight; 128-row tiles when there is too little work for them
    const int waves2 = (n_tiles2 + sm_count - 1) / sm_count;
    if (pair.status == cudaSuccess && pair.max_clusters > 0 && 2 * n_tiles2 >= sm_count && a.k_tiles >= kPairChunks && (a.row_tiles <= 1024 || a.epilogue == EPI_SWIGLU) &&
        (n_pairs + pair.max_clusters - 1) / pair.max_clusters <= waves2)
        return launch_variant<128, 1, 1, true>(a, sm_count, stream);
    return 2 * n_tiles2 >= sm_count ? launch_variant<128, 2, 1>(a, sm_count, stream) : launch_variant<128, 1, 1>(a, sm_count, stream);
}

}  // namespace

int gemm_tc_kernels(const LinearDev& lin, int64_t m, int sm_count) {
    (void)sm_count;
    return m <= 64 ? 1 : lin.w.n_bases;  // above 64 tokens one launch per basis; a k split is reduced inside the launch
}

size_t gemm_tc_act_bytes(int64_t m, int64_t k_tiles) {
    const int64_t nt = m <= 64 ? 64 : 128;
    return (size_t)((m + nt - 1) / nt * k_tiles * 4 * nt * 64);
}

// The epilogue pays where tiles follow one another and the exponentials of one are worked out under the MMAs of the next: more rounds of
// 256 x 128 tiles over the SMs the fewer MMAs a tile has.  A prefill with the quantiser's exponentials -> the epilogue's, us (two layers):
// 4096 inputs, 28672 rows, 256 tokens (1.5 rounds) 548 -> 565, 512 (3.0) 695 -> 689, 2048 (12) 1 576 -> 1 506; 3072 -> 16384, 1536 tokens
// (5.2) 835 -> 840, 2048 (6.9) 1 038 -> 1 024; 2048 -> 11264, 3072 tokens (7.1) 976 -> 980, 4096 (9.5) 1 184 -> 1 180, 8192 (19) 2 385 ->
// 2 337; 1024 -> 16384, 8192 tokens (28) 1 561 -> 1 694.
int64_t gemm_tc_swiglu_from(const LinearDev& lin, int sm_count) {
    if (lin.w.n_bases != 1 || lin.w.n_out % kTileRows != 0 || lin.w.k_tiles < 8) return INT64_MAX;
    const int64_t rounds = lin.w.k_tiles >= 16 ? 2 : (lin.w.k_tiles >= 12 ? 6 : 9), row_sets = (lin.w.row_tiles + 15) / 16;
    const int64_t blocks = (rounds * sm_count + row_sets - 1) / row_sets;  // of 128 tokens
    return std::max<int64_t>((blocks - 1) * 128 + 1, 65);
}

cudaError_t launch_gemm_tc(const LinearDev& lin, const void* x, int64_t x_stride, int64_t m, int8_t* qtc, float* sx,
                           int32_t* qsum, void* out, int64_t out_stride, int epilogue, unsigned int* err, int sm_count,
                           cudaStream_t stream, bool prequantised, bt_dtype x_dtype, float* sum) {
    if (lin.w.n_bases != 1 && epilogue == EPI_BF16 && !sum) return cudaErrorInvalidValue;
    const int nt = m <= 64 ? 64 : 128;
    if (epilogue != EPI_I32 && epilogue != EPI_F32 && epilogue != EPI_F32_ACCUM && epilogue != EPI_BF16 &&
        !(epilogue == EPI_SWIGLU && m >= gemm_tc_swiglu_from(lin, sm_count)))
        return cudaErrorInvalidValue;
    const int k = (int)lin.w.k_in, kts = (int)lin.w.k_tiles;
    cudaError_t e = cudaSuccess;
    if (prequantised) {
    } else if (x_dtype == BT_BF16) {
        e = launch_row_quant_bf16(reinterpret_cast<const __nv_bfloat16*>(x), x_stride, (int)m, k, sx, qsum, stream, qtc, kts);
    } else {
        // f32 rows: the row kernel of the decode step (identity transform); rows of a partly filled token block
        // keep whatever they held, their output columns are never stored
        e = launch_row_quant(PRE_NONE, reinterpret_cast<const float*>(x), x_stride, nullptr, 0.0f, (int)m, k, nullptr, 0, sx, qsum,
                             nullptr, stream, qtc, kts);
    }
    if (e != cudaSuccess) return e;
    // Up to 64 tokens the bases of a product are one launch: three launches in turn took 9 us each for 16 x 4096 -> 4096, of
    // which most is start-up and drain; the call 28.7 -> 18.5 us.  (Larger products fill the GPU one by one.)
    const bool together = nt == 64 && lin.w.n_bases > 1 && (epilogue == EPI_F32 || epilogue == EPI_BF16);
    for (int b = 0; b < (together ? 1 : lin.w.n_bases); ++b) {
        TcArgs a = {};
        a.bases = together ? lin.w.n_bases : 1;
        a.basis_bytes = lin.w.basis_stride();
        a.sum = sum;
        a.tiles = lin.w.tiles + (size_t)b * lin.w.basis_stride();
        a.row_tiles = lin.w.row_tiles;
        a.k_tiles = lin.w.k_tiles;
        a.n_out = lin.w.n_out;
        a.qtc = qtc;
        a.qsum = qsum;
        a.sx = sx;
        a.sw_tiles = lin.scale_tiles + (size_t)b * lin.w.row_tiles * 2;
        a.m = (int)m;
        // Several bases: the first stores, the others add to it, in basis order.  With a bf16 output all but the last work
        // on f32 rows aside, and the last one rounds the whole sum.
        const bool aside = !together && lin.w.n_bases > 1 && epilogue == EPI_BF16, last = b + 1 == lin.w.n_bases;
        a.out = aside && !last ? (void*)sum : out;
        a.out_stride = out_stride;
        a.epilogue = aside ? (last ? kEpiBf16Accum : (b > 0 ? EPI_F32_ACCUM : EPI_F32)) : ((b > 0 && epilogue == EPI_F32) ? EPI_F32_ACCUM : epilogue);
        a.acc_in = aside ? sum : reinterpret_cast<const float*>(out);
        a.err = err;
        e = launch_product(a, nt, sm_count, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace bt

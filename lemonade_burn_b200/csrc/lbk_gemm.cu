// Prefill GEMM (more than 16 token rows): int8 activations x packed ternary weights on the
// 5th-generation tensor cores (tcgen05.mma kind::i8, accumulators AND the weight operand in TMEM).
//
// Replaces ternary_gemm_multi's prefill branch and the AVX-512 register tile under it
// (crates/lb-ternary/src/gemm.rs:155-194, 245-268, 483-550).
//
// Orientation: the 128 weight rows of a tile are the MMA's M side, NT token rows its N side
// (D[row][token] in TMEM). Per 128-column block of K (one packed 32-byte block per weight row):
//
//   2 TMA threads  int8 activations [NT tok][128 B] (SWIZZLE_128B, the K-major B operand) and
//                  packed weights [128 rows][128 B] (four K blocks a box) into shared-memory rings
//                  of their own
//   2 x 4 expander thread r owns weight row r = TMEM lane r: 32 packed bytes -> 32 words of u8
//   warps          codes, word c = columns 4c..4c+3 = (packed word >> 2k) & 0x03030303; the two
//                  sets of four warps take the groups of K blocks in turn
//                  (pack.rs:10-13: no shuffles), written straight to TMEM with tcgen05.st.
//                  The expanded tile never touches shared memory: the MMAs' reads of the activations, the TMA's
//                  writes of them and 16 KB of codes a block written and read would be more than
//                  its 128 bytes a cycle.
//   MMA warp       4 x tcgen05.mma a block (A from TMEM, u8; B from shared memory, s8; K = 32 each), issued by
//                  one elected lane; tcgen05.commit frees the rings / publishes the accumulator
//   8 epilogue     tcgen05.ld, dot = acc - sum(q) (codes are w+1: gemm.rs:6-9,306-308),
//   warps          y = (float)dot * (1/(s_a*s_w)) (gemm.rs:158,178); a warp's 32 lanes are 32
//                  consecutive weight rows, so every store instruction writes 128 contiguous bytes. Two warps a
//                  quadrant of lanes, 16 token rows at a time: with one, what it computes and the stores it waits for came one after
//                  the other, 9700 cycles a tile of 192 token rows and 2000 around them, more than the tile's products; now 4400.
//
// TMEM columns: two accumulators of NT columns (the epilogue of one tile overlaps the MMAs of the
// next) + a ring of 32-column weight tiles, two hand-off groups deep at NT = 192 (4 tiles), three at NT = 64 (12).
// Bound: int8 tensor pipe; 2*m*rows*cols ops. A block of 192 token rows is 384 cycles of MMAs and takes 417 without an epilogue, 475
// beside one (585 when four epilogue warps and one-lane issue bounded it). Quantiser and GEMM, us, before -> now: 2560 -> 2 x 6912 at 17 / 333 / 2048 rows 10.4 -> 7.6,
// 20.3 -> 17.3, 74.8 -> 61.9; 6912 -> 2560 at 333 rows 17.9 -> 13.8; 4096 -> 2 x 14336 at 17 / 400 rows 19.0 -> 13.8, 51.1 -> 42.7.
#include "lbk_internal.cuh"
#include "lbk_ptx.cuh"
#include "lbk_tcgen05.cuh"

namespace lbk {

namespace {

constexpr int kBMW = 128;          // weight rows per tile (MMA M, TMEM lanes)
constexpr int kBK = 128;           // columns per stage = one packed block
constexpr int kPackBlocks = 4;      // K-blocks per packed-weight stage: [128 rows][128 B] boxes
constexpr int kPackBytes = kBMW * kBlockBytes * kPackBlocks;  // 16 KB, SWIZZLE_128B
constexpr int kEpiWarps = 8, kExpWarps = 4, kExpSets = 2;
constexpr int kEpiThreads = kEpiWarps * 32, kEpiSets = kEpiWarps / 4;
constexpr int kEpiCols = 16;      // token rows an epilogue warp takes at a time
// warps 0-7 epilogue, 8-11 and 12-15 expanders (warp % 4 = the TMEM lane quadrant a warp may touch)
// warp 16 feeds the activation ring, warp 18 the packed-weight ring: two threads, so that the weight
// stream from HBM runs ahead by its own ring's depth whatever the activation ring is waiting for
constexpr int kExpWarp0 = kEpiWarps, kTmaWarp = kExpWarp0 + kExpWarps * kExpSets, kMmaWarp = kTmaWarp + 1, kPackWarp = kTmaWarp + 2;
constexpr int kThreads = (kPackWarp + 1) * 32;
constexpr uint32_t kTmemCols = 512;
constexpr int kWide = 192;         // token rows of the wide form's tile at most
constexpr int kPlain = 0, kScatter = 1, kGated = 2;  // what the epilogue does with a tile

template <int NT>  // capacity in token rows per tile (MMA N): 192 or 64; a launch uses nt <= NT
struct Cfg {
    static constexpr int kActBytes = NT * kBK;                  // multiple of 1024 for NT = 192, 64
    static constexpr int kLoadStages = NT == kWide ? 6 : 12;    // activation ring, in K blocks
    static constexpr int kGroup = NT == kWide ? 2 : 4;          // K blocks per hand-off (see kBarFull below)
    static constexpr int kGroupStages = kLoadStages / kGroup;   // activation ring in hand-off units
    static constexpr int kAGroups = NT == kWide ? 2 : 3;        // groups of expanded weight tiles in TMEM (32 columns a tile)
    // Packed-weight ring, 16 KB a stage. With 64 token rows the weights come straight from HBM (no
    // other token tile shares them through L2) and the ring has to cover the memory latency.
    static constexpr int kPackStages = NT == kWide ? 3 : 8;
    static constexpr uint32_t kPack0 = kLoadStages * kActBytes;
    static constexpr uint32_t kAcc0 = 0, kAcc1 = NT, kA0 = 2 * NT;  // TMEM column map: two accumulators, then the weight tiles
    static_assert(2 * NT + kAGroups * kGroup * 32 <= 512, "TMEM budget");
    static constexpr int kStageGroups = kPackBlocks / kGroup;  // groups of a packed-weight stage: the second set's is the second, or every other stage's
    static_assert(kStageGroups == 1 || kStageGroups == kExpSets, "a group is half a packed-weight stage or a whole one");
    // instruction descriptor without N: D s32, A u8 (codes, TMEM), B s8 (activations), K-major, M=128
    static constexpr uint32_t kIdesc = (2u << 4) | (0u << 7) | (1u << 10) | ((kBMW >> 4) << 24);
    static constexpr uint32_t kBars = kPack0 + kPackStages * kPackBytes;
    static constexpr uint32_t kMisc = kBars + 48 * 8;
    static constexpr uint32_t kTok = kMisc + 64;              // per-token sum(q) and 1/(s_a*s_w), kGated: of gate and of up: 3 x [2][NT]
    static constexpr uint32_t kTotal = kTok + 3 * 2 * NT * 4;
    // Hand-off is by GROUPS of kGroup K blocks: a turn of the MMA warp (wait, issue, commit) takes some 330 cycles beside
    // the MMAs, as much as those of one block, so a group is 2 blocks of 192 token rows (one block a turn: 555 cycles a block) or 4 of 64. One
    // "full" barrier per group collects both operands: the activation bytes of its blocks (TMA transaction count) and one
    // arrival from each of the four expander warps whose set the group is. One "consumed" barrier per group (a single
    // tcgen05.commit) releases the activation stages and the TMEM weight slots.
    static constexpr int kBarFull = 0;                        // [group stages]
    static constexpr int kBarConsumed = kLoadStages;          // [group stages]
    static constexpr int kBarFullPack = 2 * kLoadStages;      // [PS] packed weights landed
    static constexpr int kBarEmptyPack = kBarFullPack + kPackStages;  // [PS] expanders are done with them
    static constexpr int kBarAccFull = kBarEmptyPack + kPackStages;   // [2]
    static constexpr int kBarAccEmpty = kBarAccFull + 2;      // [2]
    static_assert(kBarAccEmpty + 2 <= 48, "barrier area too small");
    static_assert(kTotal + 1024 <= 232448, "shared memory budget");
    static_assert(kAGroups <= kGroupStages, "a consumed-barrier phase must still be observable when its weight slots are filled again");
};

struct GemmParams {
    CUtensorMap act;                    // int8 [m][kp], box [NT][128], SWIZZLE_128B
    CUtensorMap wpk[LBK_MAX_GROUP];     // u8 [rows][rb], box [128][128], SWIZZLE_128B
    float *out[LBK_MAX_GROUP];
    int32_t *iout[LBK_MAX_GROUP];
    float wscale[LBK_MAX_GROUP];
    int rows[LBK_MAX_GROUP];
    int row_end[LBK_MAX_GROUP];         // running count of 128-row tiles up to and including matrix i
    int n_mat, m, m_tiles, k_blocks, total_tiles;
    int nt;                             // token rows per tile in this launch (multiple of 16, <= capacity)
    int ksplit, kb_part;                // every tile's K blocks are cut into ksplit parts of kb_part blocks (a multiple of 4)
    int32_t *acc[LBK_MAX_GROUP];        // ksplit > 1: zeroed int32 [m][rows] that the parts add their sums into
    const float *qscale;
    const int32_t *qsum;
    int *err_word;
    // matrix 0's int32 dots by token owner (see GroupArgs): rows of scatter_mt tokens per owner
    int32_t *scatter[8];
    int scatter_world, scatter_mt;
};

using namespace tc;

// A operand from TMEM (u8 codes), B from shared memory (s8 activations).
// The four K = 32 steps of one 128-column block in one go: A advances 8 TMEM columns and B 32
// bytes (2 descriptor units) per step; only the first step may start a fresh accumulator.
__device__ __forceinline__ void umma_i8_ts_block(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate_first) {
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        ".reg .b64 b1, b2, b3;\n"
        ".reg .b32 a1, a2, a3;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "setp.eq.b32 q, 0, 0;\n"
        "add.u64 b1, %2, 2;\n"
        "add.u64 b2, %2, 4;\n"
        "add.u64 b3, %2, 6;\n"
        "add.u32 a1, %1, 8;\n"
        "add.u32 a2, %1, 16;\n"
        "add.u32 a3, %1, 24;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [a1], b1, %3, q;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [a2], b2, %3, q;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [a3], b3, %3, q;\n"
        "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate_first)
        : "memory");
}
// EPI, an instantiation of its own each, so that the ordinary kernel's epilogue keeps its registers:
//   kScatter  matrix 0's int32 dots go to the token owners' buffers (GemmParams::scatter) instead of iout
//   kGated    matrices 0 and 1 are gate and up of one feed-forward, out[0] gets relu(gate)^2 * up: a tile is 64 rows of each, 16 of gate and 16 of up in turn,
//             so that a lane and the lane 16 further on hold the two factors. Half the bytes leave the kernel (2011 rows of 2560 -> 2 x 6912: 57 -> 54 us) and
//             the norm behind it reads half as many (32 -> 17 us, both in a prompt's stream). Same bits as the two projections and lbk_relu2_mul.
template <int NT, int EPI>
__global__ void __launch_bounds__(kThreads, 1) gemm_kernel(const __grid_constant__ GemmParams p) {
    using C = Cfg<NT>;
    constexpr int G = C::kGroup, PG = C::kGroupStages, PS = C::kPackStages;
    static_assert(kExpSets == 2 && kPackBlocks == 4, "the group hand-off assumes these");
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = ptx::smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *sm = smem_raw + (base - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t bar0 = base + C::kBars;
    volatile uint32_t *s_tmem = reinterpret_cast<volatile uint32_t *>(sm + C::kMisc);
    volatile int *s_abort = reinterpret_cast<volatile int *>(sm + C::kMisc + 4);
    auto bar = [&](int idx) { return bar0 + idx * 8; };

    if (tid == 0) {
        for (int i = 0; i < PG; ++i) {
            ptx::mbar_init(bar(C::kBarFull + i), 1 + kExpWarps);
            ptx::mbar_init(bar(C::kBarConsumed + i), 1);
        }
        for (int i = 0; i < PS; ++i) {
            ptx::mbar_init(bar(C::kBarFullPack + i), 1);
            ptx::mbar_init(bar(C::kBarEmptyPack + i), kExpWarps * C::kStageGroups);
        }
        for (int a = 0; a < 2; ++a) {
            ptx::mbar_init(bar(C::kBarAccFull + a), 1);
            ptx::mbar_init(bar(C::kBarAccEmpty + a), kEpiWarps);
        }
        *s_abort = 0;
        ptx::fence_barrier_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(base + C::kMisc, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem;
    // When the launch was programmatic, everything above overlapped the tail of the kernel before
    // this one (the quantiser that produces this kernel's activations). The roles that read its
    // results or write what it may still read (activation loads, epilogue) wait for it below; the
    // packed weights are constants, and their loads start at once. The kernel behind this one may be
    // scheduled as blocks of this one retire (it orders itself with its own wait).
    ptx::pdl_trigger();

    const int k_blocks = p.k_blocks;
    bool ok = true;
    // tile -> (matrix, weight-row tile, token tile); token tiles vary fastest so that CTAs running side by side share the same
    // packed weights in L2; the shorter last token tiles of a ragged batch come after all others.
    const int row_tiles = p.row_end[p.n_mat - 1], full = p.m / p.nt;
    auto decode_tile = [&](int tile, int &mat, int &m_tile, int &n_tile) {
        if (tile < full * row_tiles) {
            n_tile = tile / full;
            m_tile = tile - n_tile * full;
        } else {
            n_tile = tile - full * row_tiles;
            m_tile = full;
        }
        mat = 0;
        while (mat < p.n_mat - 1 && n_tile >= p.row_end[mat]) ++mat;
        if (mat) n_tile -= p.row_end[mat - 1];
    };

    // A work item is one tile, or one of the ksplit equal parts of a tile's K blocks. All roles walk the same items, every
    // other round backwards: a CTA whose item of the round before last was a short one gets one of those that are left over.
    const int total_items = p.total_tiles * p.ksplit, ctas = gridDim.x;
    auto item_at = [&](int round) { return round * ctas + ((round & 1) ? ctas - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x)); };
    auto item_range = [&](int item, int &tile, int &kb0, int &kb1) {
        tile = item / p.ksplit;
        const int part = item - tile * p.ksplit;
        kb0 = part * p.kb_part;
        kb1 = kb0 + p.kb_part < k_blocks ? kb0 + p.kb_part : k_blocks;
    };

    if (warp == kPackWarp) {
        // ================= TMA producer: packed weights =================
        if (lane == 0) {
            int pit = 0;
            for (int turn = 0, item; (item = item_at(turn)) < total_items && ok; ++turn) {
                int tile, kb0, kb1, mat, m_tile, n_tile;
                item_range(item, tile, kb0, kb1);
                decode_tile(tile, mat, m_tile, n_tile);
                for (int kb = kb0; kb < kb1; kb += kPackBlocks, ++pit) {  // kb0 is a multiple of kPackBlocks
                    const int ps = pit % PS, pround = pit / PS;
                    if (pround > 0 && !wait_bar(bar(C::kBarEmptyPack + ps), (pround - 1) & 1, s_abort)) {
                        ok = false;
                        break;
                    }
                    ptx::mbar_arrive_expect_tx(bar(C::kBarFullPack + ps), kPackBytes);
                    if constexpr (EPI == kGated) {
                        for (int i = 0; i < 8; ++i)
                            ptx::tma_load_2d(base + C::kPack0 + ps * kPackBytes + i * 16 * 128, &p.wpk[i & 1], bar(C::kBarFullPack + ps), kb * kBlockBytes,
                                             n_tile * (kBMW / 2) + (i >> 1) * 16);
                    } else {
                        ptx::tma_load_2d(base + C::kPack0 + ps * kPackBytes, &p.wpk[mat], bar(C::kBarFullPack + ps), kb * kBlockBytes, n_tile * kBMW);
                    }
                }
            }
        }
    } else if (warp == kTmaWarp) {
        // ================= TMA producer: activations =================
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int gr = 0;  // groups of activation blocks
            for (int turn = 0, item; (item = item_at(turn)) < total_items && ok; ++turn) {
                int tile, kb0, kb1, mat, m_tile, n_tile;
                item_range(item, tile, kb0, kb1);
                decode_tile(tile, mat, m_tile, n_tile);
                for (int kb = kb0; kb < kb1; kb += G, ++gr) {
                    const int s = gr % PG, round = gr / PG;
                    if (round > 0 && !wait_bar(bar(C::kBarConsumed + s), (round - 1) & 1, s_abort)) {
                        ok = false;
                        break;
                    }
                    const int nblk = kb1 - kb < G ? kb1 - kb : G;
                    ptx::mbar_arrive_expect_tx(bar(C::kBarFull + s), static_cast<uint32_t>(nblk * p.nt) * kBK);
                    for (int b = 0; b < nblk; ++b)
                        ptx::tma_load_2d(base + (s * G + b) * C::kActBytes, &p.act, bar(C::kBarFull + s), (kb + b) * kBK, m_tile * p.nt);
                }
            }
        }
    } else if (warp >= kExpWarp0 && warp < kExpWarp0 + kExpWarps * kExpSets) {
        // ================= expanders: packed 2-bit -> u8 codes in TMEM =================
        // The sets take the groups of K blocks in turn: the codes of two blocks are worked out in registers while the slots they go to are
        // still being read, so what lies between a slot that is free again and its next "full" is one store and its wait. With
        // a block of every group for each set, the set's own turn (waits, arrivals, a store of 250 cycles a block) bounded the kernel.
        const int quad = (warp - kExpWarp0) % kExpWarps, set = (warp - kExpWarp0) / kExpWarps;
        const int r = quad * 32 + lane;  // weight row of the tile = TMEM lane
        const uint32_t a_dst = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + C::kA0;
        const uint8_t *pk_row = sm + C::kPack0 + r * 128;  // row r of a [128][128 B] swizzled stage; block b's 32 bytes are units 2 b, 2 b + 1
        const int x = r & 7;
        int gr = 0, stage = 0;  // groups and packed-weight stages so far
        for (int turn = 0, item; (item = item_at(turn)) < total_items && ok; ++turn) {
            int tile, kb0, kb1;
            item_range(item, tile, kb0, kb1);
            for (int kb = kb0; kb < kb1; kb += kPackBlocks, ++stage) {
                const int groups = C::kStageGroups == 1 || kb + G >= kb1 ? 1 : 2;  // of this stage
                const int mine = C::kStageGroups == 1 ? gr : gr + set;               // the number of this set's
                const bool have = C::kStageGroups == 1 ? (gr & 1) == set : set < groups;
                gr += groups;
                if (C::kStageGroups == 1 && !have) continue;
                const int ps = stage % PS;
                if (!warp_wait(bar(C::kBarFullPack + ps), (stage / PS) & 1, s_abort)) {
                    ok = false;
                    break;
                }
                if (!have) {  // a last stage without a group of this set goes by
                    if (lane == 0) ptx::mbar_arrive(bar(C::kBarEmptyPack + ps));
                    continue;
                }
                const uint8_t *pk = pk_row + ps * kPackBytes;
#pragma unroll
                for (int half = 0; half < G / 2; ++half) {
                    const int u0 = 4 * (C::kStageGroups == 1 ? half : set);  // first of the two blocks' four units
                    uint32_t v[64];  // word 32 b + 8 k + i = columns k * 32 + 4 i .. 4 i + 3 of block b (blocks behind the end are not read)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const uint4 w4 = *reinterpret_cast<const uint4 *>(pk + (((u0 + u) ^ x) << 4));  // packed bytes 16 (u % 2) .. of block u / 2
                        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
#pragma unroll
                            for (int i = 0; i < 4; ++i) v[32 * (u / 2) + 8 * k + 4 * (u % 2) + i] = (w[i] >> (2 * k)) & 0x03030303u;
                    }
                    if (half == 0) {
                        // these TMEM slots were last read by group mine - kAGroups
                        const int last = mine - C::kAGroups;
                        if (last >= 0 && !warp_wait(bar(C::kBarConsumed + last % PG), (last / PG) & 1, s_abort)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                    }
                    tmem_st64(a_dst + ((mine % C::kAGroups) * G + 2 * half) * 32, v);
                }
                if (!ok) break;
                // The stage is given back behind the stores: what they take has arrived from shared memory. Given back as soon as the loads were
                // issued, it was filled again, once in some thousand tiles, before a load behind the epilogue's stores had read its first rows.
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar(C::kBarEmptyPack + ps));
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar(C::kBarFull + mine % PG));
            }
        }
    } else if (warp == kMmaWarp) {
        // ================= MMA issuer =================
        // The whole warp walks and waits, one elected lane issues.
        int tcount = 0, sp = 0, as = 0;
        uint32_t full_phase = 0;
        const uint64_t bdesc0 = smem_desc_sw128(base);  // activation block stage 0; stage s adds s * kActBytes / 16
        for (int item; (item = item_at(tcount)) < total_items; ++tcount) {
            const int a = tcount & 1, around = tcount >> 1;
            if (around > 0) ok = warp_wait(bar(C::kBarAccEmpty + a), (around - 1) & 1, s_abort) && ok;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (a ? C::kAcc1 : C::kAcc0);
            // N of this tile: the launch's token tile, less for the last tile of a ragged batch
            int tile, kb0, kb1, mat, m_tile, n_tile;
            item_range(item, tile, kb0, kb1);
            decode_tile(tile, mat, m_tile, n_tile);
            const int left = p.m - m_tile * p.nt;
            const int n_mma = left < p.nt ? (left + 15) & ~15 : p.nt;
            const uint32_t idesc = C::kIdesc | (static_cast<uint32_t>(n_mma >> 3) << 17);
            for (int kb = kb0; kb < kb1; kb += G) {
                ok = warp_wait(bar(C::kBarFull + sp), full_phase, s_abort) && ok;
                tc_fence_after();
                const uint32_t a_tmem = tmem_base + C::kA0 + as * (G * 32);
                const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(sp * G * (C::kActBytes >> 4));
                if (elect_one() && ok) {
                    umma_i8_ts_block(d_tmem, a_tmem, bdesc, idesc, kb != kb0 ? 1u : 0u);
#pragma unroll
                    for (int b = 1; b < G; ++b)
                        if (kb + b < kb1) umma_i8_ts_block(d_tmem, a_tmem + b * 32, bdesc + static_cast<uint64_t>(b * (C::kActBytes >> 4)), idesc, 1u);
                    umma_commit(bar(C::kBarConsumed + sp));  // both operands' slots are reusable once these MMAs retire
                    if (kb + G >= kb1) umma_commit(bar(C::kBarAccFull + a));  // accumulator complete
                }
                __syncwarp();
                if (++sp == PG) {
                    sp = 0;
                    full_phase ^= 1u;
                }
                if (++as == C::kAGroups) as = 0;
            }
        }
    } else if (warp < kEpiWarps) {
        // ================= epilogue (warp % 4 = TMEM lane quadrant) =================
        int *s_qs = reinterpret_cast<int *>(sm + C::kTok);
        float *s_inv = reinterpret_cast<float *>(sm + C::kTok + 2 * NT * 4), *s_inv2 = s_inv + 2 * NT;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // Per-token terms of a tile: a thread asks for those of tokens tid and tid + 128 one tile ahead, before this tile's stores. One warp that
        // fetched them 32 at a time in front of the tile held the accumulators for 5500 of the 14400 cycles a tile of 2560 columns took. Calls with
        // small tiles have one or two a CTA, their terms come during the products: warp 0 fetches them there (ahead it was 1 us slower at 333 rows).
        constexpr bool kAhead = NT > 128;
        constexpr int kTerms = (NT + kEpiThreads - 1) / kEpiThreads;
        const int quad = warp & 3;
        int term_q[kTerms];
        float term_s[kTerms];
        auto fetch_terms = [&](int item) {
            if (item >= total_items) return;
            int tile, kb0, kb1, mat, m_tile, n_tile;
            item_range(item, tile, kb0, kb1);
            decode_tile(tile, mat, m_tile, n_tile);
#pragma unroll
            for (int e = 0; e < kTerms; ++e) {
                const int i = tid + e * kEpiThreads, tk = m_tile * p.nt + i;
                const bool in = i < p.nt && tk < p.m;
                term_q[e] = in ? p.qsum[tk] : 0;
                term_s[e] = in && p.qscale ? p.qscale[tk] : 0.0f;
            }
        };
        if constexpr (kAhead) fetch_terms(item_at(0));
        int tcount = 0;
        for (int item; (item = item_at(tcount)) < total_items && ok; ++tcount) {
            const int a = tcount & 1, around = tcount >> 1;
            int tile, kb0, kb1, mat, m_tile, n_tile;
            item_range(item, tile, kb0, kb1);
            decode_tile(tile, mat, m_tile, n_tile);
            const int rows = p.rows[mat];
            const int row = EPI == kGated ? n_tile * (kBMW / 2) + quad * 16 + (lane & 15) : n_tile * kBMW + quad * 32 + lane;
            const int nt = p.nt;
            const int tok0 = m_tile * nt;
            float *out = p.out[mat];
            int32_t *iout = p.iout[mat];
            int *qs = s_qs + a * NT;  // reuse by accumulator parity is safe: see acc_empty below
            float *inv = s_inv + a * NT, *inv2 = s_inv2 + a * NT;
            if constexpr (kAhead) {
#pragma unroll
                for (int e = 0; e < kTerms; ++e) {
                    const int i = tid + e * kEpiThreads, tk = tok0 + i;
                    if (i < NT) {
                        qs[i] = term_q[e];
                        inv[i] = i < nt && tk < p.m && p.qscale ? __fdiv_rn(1.0f, __fmul_rn(term_s[e], p.wscale[mat])) : 0.0f;  // gemm.rs:158
                        if constexpr (EPI == kGated) inv2[i] = i < nt && tk < p.m ? __fdiv_rn(1.0f, __fmul_rn(term_s[e], p.wscale[1])) : 0.0f;
                    }
                }
                fetch_terms(item_at(tcount + 1));
            } else if (warp == 0) {
                for (int i = lane; i < nt; i += 32) {
                    const int tk = tok0 + i;
                    qs[i] = tk < p.m ? p.qsum[tk] : 0;
                    inv[i] = (tk < p.m && p.qscale) ? __fdiv_rn(1.0f, __fmul_rn(p.qscale[tk], p.wscale[mat])) : 0.0f;  // gemm.rs:158
                    if constexpr (EPI == kGated) inv2[i] = tk < p.m ? __fdiv_rn(1.0f, __fmul_rn(p.qscale[tk], p.wscale[1])) : 0.0f;
                }
            }
            ptx::named_barrier(2, kEpiThreads);  // the epilogue warps
            if (!warp_wait(bar(C::kBarAccFull + a), around & 1, s_abort)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const int ntok = p.m - tok0 < nt ? p.m - tok0 : nt;
#pragma unroll 1
            for (int c = warp >> 2; c * kEpiCols < ntok; c += kEpiSets) {
                uint32_t v[kEpiCols];
                tmem_ld16(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + (a ? C::kAcc1 : C::kAcc0) + c * kEpiCols, v);
                // per-token terms into registers first: the stores below may alias the shared
                // arrays as far as the compiler knows, which would serialise load -> store pairs
                int q[kEpiCols];
                float sc[kEpiCols];
#pragma unroll
                for (int i = 0; i < kEpiCols; i += 4) {
                    const int4 q4 = *reinterpret_cast<const int4 *>(qs + c * kEpiCols + i);
                    const float4 s4 = *reinterpret_cast<const float4 *>((EPI == kGated && lane >= 16 ? inv2 : inv) + c * kEpiCols + i);
                    q[i] = q4.x; q[i + 1] = q4.y; q[i + 2] = q4.z; q[i + 3] = q4.w;
                    sc[i] = s4.x; sc[i + 1] = s4.y; sc[i + 2] = s4.z; sc[i + 3] = s4.w;
                }
                tmem_ld_wait();
                if constexpr (EPI == kScatter) {
                    // The reduce-scatter of a row-parallel layer starts here: the int32 dots of a token go straight
                    // into the buffer of the rank that owns the token (plain stores into peer memory, 128 consecutive
                    // bytes per warp instruction), while the MMAs of the next tile run.
                    if (row < rows) {
                        const int tk = tok0 + c * kEpiCols;
                        int o = tk / p.scatter_mt, lt = tk - o * p.scatter_mt;
#pragma unroll
                        for (int i = 0; i < kEpiCols; ++i) {
                            if (c * kEpiCols + i < ntok) p.scatter[o][static_cast<size_t>(lt) * rows + row] = static_cast<int>(v[i]) - q[i];
                            if (++lt == p.scatter_mt) {
                                lt = 0;
                                ++o;
                            }
                        }
                    }
                    continue;
                }
                if constexpr (EPI == kGated) {
                    // of two token rows in turn the lower half of the warp finishes the first and the upper half the second
                    const bool up = lane >= 16;
#pragma unroll
                    for (int i = 0; i < kEpiCols; i += 2) {
                        const float y0 = __fmul_rn(__int2float_rn(static_cast<int>(v[i]) - q[i]), sc[i]), y1 = __fmul_rn(__int2float_rn(static_cast<int>(v[i + 1]) - q[i + 1]), sc[i + 1]);
                        const float other = __shfl_xor_sync(0xffffffffu, up ? y0 : y1, 16), gate = fmaxf(up ? other : y0, 0.0f), by = up ? y1 : other;
                        const int tk = c * kEpiCols + i + (up ? 1 : 0);
                        if (row < rows && tk < ntok) out[static_cast<size_t>(tok0 + tk) * rows + row] = __fmul_rn(__fmul_rn(gate, gate), by);
                    }
                    continue;
                }
                if (p.ksplit > 1) {
                    // one of several parts of this tile: add the sums into the zeroed int32 buffer
                    // (the part that starts at block 0 also takes off sum(q)); a small kernel scales later
                    if (row < rows) {
                        int32_t *dst = p.acc[mat] + static_cast<size_t>(tok0 + c * kEpiCols) * rows + row;
#pragma unroll
                        for (int i = 0; i < kEpiCols; ++i)
                            if (c * kEpiCols + i < ntok) atomicAdd(dst + static_cast<size_t>(i) * rows, static_cast<int>(v[i]) - (kb0 == 0 ? q[i] : 0));
                    }
                    continue;
                }
                if (row < rows) {
                    const size_t o0 = static_cast<size_t>(tok0 + c * kEpiCols) * rows + row;
                    if (c * kEpiCols + kEpiCols <= ntok) {
                        if (out) {
#pragma unroll
                            for (int i = 0; i < kEpiCols; ++i)
                                out[o0 + static_cast<size_t>(i) * rows] = __fmul_rn(__int2float_rn(static_cast<int>(v[i]) - q[i]), sc[i]);
                        }
                        if (iout) {
#pragma unroll
                            for (int i = 0; i < kEpiCols; ++i) iout[o0 + static_cast<size_t>(i) * rows] = static_cast<int>(v[i]) - q[i];
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < kEpiCols; ++i) {
                            if (c * kEpiCols + i < ntok) {
                                const int d = static_cast<int>(v[i]) - q[i];
                                if (iout) iout[o0 + static_cast<size_t>(i) * rows] = d;
                                if (out) out[o0 + static_cast<size_t>(i) * rows] = __fmul_rn(__int2float_rn(d), sc[i]);
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            ptx::named_barrier(2, kEpiThreads);  // all epilogue warps are done with qs/inv of this parity
            if (lane == 0) ptx::mbar_arrive(bar(C::kBarAccEmpty + a));
        }
    }

    if (!ok && lane == 0) atomicExch(p.err_word, 5);
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace

template <int NT>
static int init_one(Ctx *ctx) {
    const size_t smem = Cfg<NT>::kTotal + 1024;
    if (smem > ctx->smem_optin) return fail(LBK_ERR_UNSUPPORTED, "gemm kernel needs %zu B of shared memory", smem);
    for (void (*k)(GemmParams) : {gemm_kernel<NT, kPlain>, gemm_kernel<NT, kScatter>, gemm_kernel<NT, kGated>})
        LBK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    return LBK_OK;
}

int gemm_init(Ctx *ctx) {
    LBK_TRY(init_one<kWide>(ctx));
    LBK_TRY(init_one<64>(ctx));
    LBK_CUDA(cudaMalloc(&ctx->gemm_acc, kGemmAccBytes));
    LBK_CUDA(cudaMemset(ctx->gemm_acc, 0, kGemmAccBytes));  // kept zero between launches: the scaling kernel zeroes what it reads
    return LBK_OK;
}
static const InitHook kInitGemm(gemm_init);

// Token rows per tile for a launch, a multiple of 16, and parts to cut every tile's K blocks into: the pair with the least cost in cycles of the fullest CTA.
// A K block takes 250 cycles in the narrow kernel, which runs up to 64 token rows; in the wide one 365 at 96 and 490 at 192 (launches of many
// rounds, their epilogues beside the products; 341 and 416 in a single round). 15 cycles a token row are the last tile's
// epilogue, 300 the start of a tile. Short tiles of a ragged batch come last (decode_tile in the kernel): what is left
// over behind the full rounds are short ones, and with the order turned round every other time a CTA that has two of them
// at the end takes less than a full tile longer than the others.
// A launch with few tiles against the SM count (small token batches, tensor-parallel shards) leaves SMs idle: parts add
// their int32 sums into a zeroed buffer, 60 cycles a token row and tile, and a small kernel scales them afterwards, 6000 cycles, and 0.004 for each sum
// and each time it is added, read and zeroed. A cut has to be 7 % better.
// The constants are fitted to every tile and cut of 14 groups of 512 to 28672 columns at 15 sizes: the choice is 1.4 % slower than the best pair (geometric mean). Tile first
// and cut afterwards (3.3 %), with an epilogue as four warps did it and rounds counted as whole ones, had us, chosen then / now: 777 rows of 8192 -> 2 x 2048 75 / 31, 2048 of
// 512 -> 2 x 1376 16.7 / 11.9, 24 of 14336 -> 4096 17.0 / 12.4, 150 of 20480 -> 1000 20.1 / 14.9.
struct TileChoice {
    int nt = 0, ksplit = 1, kb_part = 0;
};
static TileChoice choose_tile(int m, int row_tiles, size_t rows, int k_blocks, int sms, bool may_cut) {
    auto block = [](int nt) { return nt <= 64 ? 250.0 : 240.0 + 1.3 * nt; };
    TileChoice best;
    double best_cost = 0.0;
    for (int nt = 16; nt <= kWide; nt += 16) {
        const int full = m / nt, rest = m % nt;
        const long long shorts = rest ? row_tiles : 0, tiles = static_cast<long long>(full) * row_tiles + shorts;
        const long long whole = tiles / sms, left = tiles % sms;
        const double part = full && rest ? (240.0 + 1.3 * rest) / block(nt) : 1.0, least = part < 1.0 ? part : 1.0;
        double rounds = static_cast<double>(whole);
        if (left > shorts) rounds += 1.0;
        else if (left > 0 && 2 * left <= shorts && whole > 0) rounds += 2.0 * least > 1.0 ? 2.0 * least - 1.0 : 0.0;
        else if (left > 0) rounds += least;
        const double last = 15.0 * nt, uncut = rounds * (k_blocks * block(nt) + 300.0) + last;
        if (best.nt == 0 || uncut < best_cost) {
            best_cost = uncut;
            best = {nt, 1, k_blocks};
        }
        for (int s = 2; may_cut && s <= 8; ++s) {
            const int per = ((k_blocks + s - 1) / s + kPackBlocks - 1) / kPackBlocks * kPackBlocks;
            if (per < 2 * kPackBlocks) break;
            if ((k_blocks + per - 1) / per != s) continue;  // rounding made fewer parts: that count is or was tried as itself
            const double cost = static_cast<double>((tiles * s + sms - 1) / sms) * (per * block(nt) + 300.0 + 60.0 * nt) + last + 6000.0 +
                                0.004 * m * static_cast<double>(rows) * (s + 2);
            if (cost < 0.93 * best_cost) {
                best_cost = cost;
                best = {nt, s, per};
            }
        }
        if (nt >= m) break;
    }
    return best;
}

int launch_gemm(Ctx *ctx, const GroupArgs &g, cudaStream_t stream) {
    if (!g.q || !g.qsum) return fail(LBK_ERR_INVALID, "gemm: quantised activations are required");
    if (g.n < 1 || g.n > LBK_MAX_GROUP) return fail(LBK_ERR_INVALID, "group size %d not in 1..%d", g.n, LBK_MAX_GROUP);
    if (g.m == 0) return LBK_OK;
    GemmParams p{};
    const size_t kp = g.w[0]->kp;
    int row_tiles = 0;
    if (g.gated && (g.n != 2 || g.w[0]->rows != g.w[1]->rows || g.iout[0] || g.iout[1] || g.scatter_world || !g.qscale || !g.out[0]))
        return fail(LBK_ERR_INVALID, "gemm: a gated pair is two matrices of one shape with an f32 output");
    for (int i = 0; i < g.n; ++i) row_tiles += static_cast<int>((g.w[i]->rows + kBMW - 1) / kBMW);
    if (g.gated) row_tiles = static_cast<int>((g.w[0]->rows + kBMW / 2 - 1) / (kBMW / 2));
    // A cut tile's parts meet in the caller's integer outputs where they are given, else in slices of the context's buffer. Not before a gated pair's product, and
    // not in peer memory.
    size_t rows = 0, need = 0;
    for (int i = 0; i < g.n; ++i) {
        rows += g.w[i]->rows;
        if (!g.iout[i]) need += (g.m * g.w[i]->rows * sizeof(int32_t) + 255) / 256 * 256;
    }
    const TileChoice choice = choose_tile(static_cast<int>(g.m), row_tiles, rows, static_cast<int>(kp / kBK), ctx->sm_count, !g.gated && !g.scatter_world && need <= kGemmAccBytes);
    const int nt = choice.nt;
    LBK_TRY(encode_act_map(&p.act, g.q, g.m, kp, nt));
    p.nt = nt;
    p.m = static_cast<int>(g.m);
    p.m_tiles = static_cast<int>((g.m + nt - 1) / nt);
    p.k_blocks = static_cast<int>(kp / kBK);
    row_tiles = 0;
    for (int i = 0; i < g.n; ++i) {
        const Weight *w = g.w[i];
        if (w->kp != kp) return fail(LBK_ERR_SHAPE, "inner dimension mismatch");
        if (g.out[i] && !g.qscale) return fail(LBK_ERR_INVALID, "gemm: f32 outputs need the activation scales");
        p.wpk[i] = g.gated ? w->tmap_gemv : w->tmap_gemm;  // boxes of 16 rows or of 128
        p.out[i] = g.out[i];
        p.iout[i] = g.iout[i];
        p.wscale[i] = w->scale;
        p.rows[i] = static_cast<int>(w->rows);
        row_tiles += static_cast<int>((w->rows + kBMW - 1) / kBMW);
        p.row_end[i] = row_tiles;
    }
    p.n_mat = g.n;
    if (g.gated) {  // one matrix of pairs
        p.n_mat = 1;
        p.row_end[0] = row_tiles = static_cast<int>((g.w[0]->rows + kBMW / 2 - 1) / (kBMW / 2));
    }
    const int tiles = row_tiles * p.m_tiles;
    p.total_tiles = tiles;
    p.qscale = g.qscale;
    p.qsum = g.qsum;
    p.err_word = ctx->err_word;
    if (tiles == 0 || p.k_blocks == 0) return LBK_OK;
    p.ksplit = choice.ksplit;
    p.kb_part = choice.kb_part;
    p.scatter_world = g.scatter_world;
    p.scatter_mt = g.scatter_mt;
    for (int i = 0; i < 8; ++i) p.scatter[i] = g.scatter_base[i];
    if (g.scatter_world) {
        if (g.n != 1 || g.scatter_mt < 1) return fail(LBK_ERR_INVALID, "gemm: scattered outputs take one matrix");
    }
    if (p.ksplit > 1) {
        size_t off = 0;
        for (int i = 0; i < g.n; ++i) {
            const size_t bytes = g.m * g.w[i]->rows * sizeof(int32_t);
            if (g.iout[i]) {
                p.acc[i] = g.iout[i];
                LBK_CUDA(cudaMemsetAsync(p.acc[i], 0, bytes, stream));  // the caller's buffer holds whatever it held
            } else {
                // the context's buffer is zero at rest (launch_scale_epilogue_group zeroes what it reads)
                p.acc[i] = reinterpret_cast<int32_t *>(reinterpret_cast<char *>(ctx->gemm_acc) + off);
                off += (bytes + 255) / 256 * 256;
            }
        }
    }
    const int items = tiles * p.ksplit;
    const int grid = items < ctx->sm_count ? items : ctx->sm_count;
    // programmatic stream serialisation: this grid may start while the previous kernel of the
    // stream is still draining (see griddepcontrol.wait in the kernel)
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cfg.dynamicSmemBytes = (nt > 64 ? Cfg<kWide>::kTotal : Cfg<64>::kTotal) + 1024;
    void (*kernel)(GemmParams) = nt > 64 ? gemm_kernel<kWide, kPlain> : gemm_kernel<64, kPlain>;
    if (p.scatter_world) kernel = nt > 64 ? gemm_kernel<kWide, kScatter> : gemm_kernel<64, kScatter>;
    if (g.gated) kernel = nt > 64 ? gemm_kernel<kWide, kGated> : gemm_kernel<64, kGated>;
    LBK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    LBK_CUDA(cudaGetLastError());
    ctx->launches++;
    if (p.ksplit > 1) {  // one launch scales every matrix of the group (and zeroes the context's sums again)
        int32_t *dots[LBK_MAX_GROUP];
        float *outs[LBK_MAX_GROUP];
        float ws[LBK_MAX_GROUP];
        int rows[LBK_MAX_GROUP];
        bool clean[LBK_MAX_GROUP];
        bool any = false;
        for (int i = 0; i < g.n; ++i) {
            dots[i] = p.acc[i];
            outs[i] = g.out[i];
            ws[i] = g.w[i]->scale;
            rows[i] = static_cast<int>(g.w[i]->rows);
            clean[i] = g.iout[i] == nullptr;
            any = any || g.out[i] != nullptr || clean[i];
        }
        if (any) LBK_TRY(launch_scale_epilogue_group(ctx, g.n, dots, outs, ws, rows, clean, g.qscale, g.m, stream));
    }
    return LBK_OK;
}

}  // namespace lbk

// Few tokens (up to 16) against bf16 weights: the streaming loop shared by the projections (lbk_dense.cu) and the
// experts (lbk_moe.cu). Bound: HBM, the weights once.
//
//   rows      a CTA owns a contiguous range of weight rows over the whole of K, cut into boxes of at most 32 rows whose size is chosen so that
//             all SMs have the same number of rows (2560 rows: 18 each); nothing crosses CTAs. Cutting (tile, K) runs between CTAs
//             instead was built twice: the partial sums' trip through L2 (store, fence, count, read back) cost 3 to 4 us of a 10 us kernel.
//   boxes     a box is up to 32 rows (two tiles of the product) x 64 columns, laid down by TMA with the 128-byte swizzle. The 16 warps take the
//             64-column chunks of K in turn, so that what is in flight is neighbouring memory; a warp owns a ring of boxes
//             and goes through its chunks for up to kTiles tiles at a time, so nothing in the loop crosses warps and a
//             token's values are read once for all of these tiles. Whole 128-byte lines by TMA,
//             and not 64-byte pieces by lanes, is what the rate comes from: lanes that load MMA fragments straight from
//             global memory got 1.8 to 2.4 TB/s out of weights 2560 wide and 4.7 out of 4096 -> 2 x 14336.
//   product   mma.sync m16n8k16, the tile's rows as M, tokens as N. Lane (g, t) takes 16-byte units 2t and 2t + 1 of rows
//             g and g + 8: two units are two MMAs' operands each, because the contraction index may be permuted as
//             long as weights and tokens are permuted alike. Conflict-free under the swizzle.
//   sums      the 16 warps' accumulators meet in shared memory, in warp order, once per kTiles tiles.
#pragma once

#include "lbk_dense_dev.cuh"
#include "lbk_ptx.cuh"

namespace lbk {
namespace few {

constexpr int kThreads = 512, kWarps = 16;
constexpr int kMaxTokens = 16;
constexpr int kRingBytes = 9216;            // a warp's ring: two to four boxes, each from a multiple of 1024 bytes on
constexpr int kMaxBoxes = 4;
constexpr int kTiles = 4;                   // weight tiles whose sums a warp carries at a time (gated: two of gate, two of up)
constexpr uint32_t kWaitLimit = 1u << 22;   // polls before a wait gives up

// Shared memory from a 1024-byte aligned base: rings, barriers, the warps' sums, then what the kernel adds.
__host__ __device__ constexpr int red_floats(int ntl) { return kTiles * ntl * 128; }  // of one warp
__host__ __device__ constexpr int bars_at() { return kWarps * kRingBytes; }
__host__ __device__ constexpr int red_at() { return bars_at() + kWarps * kMaxBoxes * 8; }
__host__ __device__ constexpr int rest_at(int ntl) { return red_at() + kWarps * red_floats(ntl) * 4; }

// A box's place in the ring, and how many there are.
__host__ __device__ inline int slot_bytes(int box_rows) { return (box_rows * 128 + 1023) / 1024 * 1024; }
__host__ __device__ inline int ring_depth(int box_rows) {
    const int d = kRingBytes / slot_bytes(box_rows);
    return d < kMaxBoxes ? d : kMaxBoxes;
}

// How `rows` weight rows are dealt to `sms` CTAs: `boxes` boxes of box_rows rows each, as few as there can be. A box costs its warp a wait, a refill
// and a chain of MMAs whatever its rows, and fewer, larger ones leave fewer rows over, so fewer SMs idle. (Choosing the most bytes in flight instead took,
// at one token: 4096 -> 16384 27.9 us in five boxes of 23 rows, 24.0 in four of 28; 4096 -> 2 x 9472 30.7 in three of 22, 26.6 in two of 32; 8192 -> 2 x
// 28672 171 in thirteen of 15, 135 in seven of 28; nothing measured is slower.)
struct Deal {
    int box_rows = 16, boxes = 1, ctas = 1;
};
inline Deal deal_rows(size_t rows, int sms) {
    Deal d;
    const int each = static_cast<int>((rows + sms - 1) / sms);
    d.boxes = (each + 31) / 32;
    d.box_rows = (each + d.boxes - 1) / d.boxes;
    const size_t per = static_cast<size_t>(d.boxes) * d.box_rows;
    d.ctas = static_cast<int>((rows + per - 1) / per);
    return d;
}

// how many of `chunks` chunks are warp, warp + 16, ...
__device__ __forceinline__ int chunks_of(int chunks, int warp) { return chunks > warp ? (chunks - warp + kWarps - 1) / kWarps : 0; }

__device__ __forceinline__ void prefetch_box(const CUtensorMap *map, int c0, int c1) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(c0), "r"(c1) : "memory");
}

// Units 2t and 2t + 1 of 64 columns of this lane's token of every eight.
template <int NTL>
struct Tokens {
    uint4 lo[NTL], hi[NTL];
};

// This lane's places in a box.
struct Units {
    uint32_t a, b;
    __device__ __forceinline__ explicit Units(int lane) {
        const int g = lane >> 2, t = lane & 3;
        a = g * 128 + (((2 * t) ^ g) << 4);
        b = g * 128 + (((2 * t + 1) ^ g) << 4);
    }
};

// One box (MT tiles) times the tokens' 64 columns. Rows past the box's end are whatever lies behind it; what comes of them
// is dropped with them.
template <int NTL, int MT>
__device__ __forceinline__ void box_mma(const uint8_t *st, Units u, const Tokens<NTL> &x, float (*acc)[NTL][4]) {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const uint8_t *lo = st + m * 2048, *hi = lo + 1024;
        const uint4 l0 = *reinterpret_cast<const uint4 *>(lo + u.a), l1 = *reinterpret_cast<const uint4 *>(lo + u.b);
        const uint4 h0 = *reinterpret_cast<const uint4 *>(hi + u.a), h1 = *reinterpret_cast<const uint4 *>(hi + u.b);
        const uint32_t a0[4] = {l0.x, h0.x, l0.y, h0.y}, a1[4] = {l0.z, h0.z, l0.w, h0.w};
        const uint32_t a2[4] = {l1.x, h1.x, l1.y, h1.y}, a3[4] = {l1.z, h1.z, l1.w, h1.w};
#pragma unroll
        for (int j = 0; j < NTL; ++j) {
            ptx::mma_bf16(acc[m][j], a0, x.lo[j].x, x.lo[j].y);
            ptx::mma_bf16(acc[m][j], a1, x.lo[j].z, x.lo[j].w);
            ptx::mma_bf16(acc[m][j], a2, x.hi[j].x, x.hi[j].y);
            ptx::mma_bf16(acc[m][j], a3, x.hi[j].z, x.hi[j].w);
        }
    }
}

// A warp's ring: `fetch` (lane 0) starts a box of the warp's sequence into a slot.
struct Ring {
    uint8_t *data;
    uint32_t data_addr, bar_addr;
    int slot, box_bytes, depth;
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    __device__ __forceinline__ Ring(uint8_t *sm, uint32_t base, int warp, int box_rows)
        : data(sm + warp * kRingBytes), data_addr(base + warp * kRingBytes), bar_addr(base + bars_at() + warp * (kMaxBoxes * 8)), slot(slot_bytes(box_rows)),
          box_bytes(box_rows * 128), depth(ring_depth(box_rows)) {}
    __device__ __forceinline__ void init() const {  // lane 0
        for (int i = 0; i < kMaxBoxes; ++i) ptx::mbar_init(bar_addr + i * 8, 1);
        ptx::fence_barrier_init();
    }
    __device__ __forceinline__ void fetch(int i, const CUtensorMap *map, int c0, int row) const {
        ptx::mbar_arrive_expect_tx(bar_addr + i * 8, static_cast<uint32_t>(box_bytes));
        ptx::tma_load_2d(data_addr + i * slot, map, bar_addr + i * 8, c0, row);
    }
    __device__ __forceinline__ const uint8_t *wait() {
        if (!ptx::mbar_wait(bar_addr + s * 8, phase, kWaitLimit)) ok = false;
        return data + s * slot;
    }
    __device__ __forceinline__ void next() {
        if (++s == depth) {
            s = 0;
            phase ^= 1;
        }
    }
};

template <int NTL>
__device__ __forceinline__ void zero(float (&v)[kTiles][NTL][4]) {
#pragma unroll
    for (int k = 0; k < kTiles; ++k)
#pragma unroll
        for (int j = 0; j < NTL; ++j) v[k][j][0] = v[k][j][1] = v[k][j][2] = v[k][j][3] = 0.0f;
}
// a warp's sums of `tiles` tiles, in the accumulator layout
template <int NTL>
__device__ __forceinline__ void leave(float *red, int lane, int tiles, const float (&v)[kTiles][NTL][4]) {
#pragma unroll
    for (int k = 0; k < kTiles; ++k)
        if (k < tiles) {
#pragma unroll
            for (int j = 0; j < NTL; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) red[((k * NTL + j) * 4 + i) * 32 + lane] = v[k][j][i];
        }
}
// place `f` of tile `k` over all warps
template <int NTL>
__device__ __forceinline__ float collect(const float *red, int k, int f) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v += red[w * red_floats(NTL) + k * NTL * 128 + f];
    return v;
}
// which row of its tile and which token place `f` is
__device__ __forceinline__ int place_row(int f) { return ((f & 31) >> 2) + ((f >> 6) & 1) * 8; }
__device__ __forceinline__ int place_token(int f) { return (f >> 7) * 8 + 2 * (f & 3) + ((f >> 5) & 1); }

}  // namespace few
}  // namespace lbk

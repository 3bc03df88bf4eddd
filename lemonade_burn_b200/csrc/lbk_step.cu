// A decode step of the ternary decoder in one launch: every layer's norms, projections, RoPE, cache append and attention
// (crates/lb-model/src/model.rs:305-374 with one token per sequence), for up to 16 sequences.
//
// Bound of a step: the packed weights and the cached keys and values once, from HBM. A kernel per operation is bound by something
// else: at 2560 wide a layer's projections stream 118 KB per SM, 3 us in all, but six dependent launches with their set-up,
// first loads and input rows took 43 us. Here one CTA per SM stays for the whole step (cooperative launch), and
//
//   weights     every warp owns a ring of TMA stages and a list of stages that goes on through all projections of all layers,
//               so the ring is refilled with the next projection's weights while this one waits for its input;
//   projections gemv_kernel's arithmetic (lbk_gemv_core.cuh): a CTA owns a contiguous range of 16-row tiles, its 16 warps share the
//               (tile, chunk) stages, and meet in shared memory; same integers, same scale product. Gate and up tiles lie
//               side by side, so relu(gate)^2 * up leaves as one row;
//   meetings    between dependent parts all CTAs meet on a counter in L2, 6 times a layer. The thread that arrives is the one that
//               polls: polls of other warps held the arriving thread's release up by 10000 cycles. Norm weights and cached rows are
//               asked for between arriving and waiting. A barrier, whose count is ordered behind the CTA's values, costs 2500 to 3500
//               cycles, a third of it until the values are known to be in L2. With one sequence five of the six are loose: the count
//               goes out beside the values, and a reader tells by the words themselves whether they are there (Place). A step of
//               30 layers of 2560 at 2000 positions 868 -> 822 us, of 12 layers at 100 positions 319 -> 302. With more
//               sequences, whose rows one CTA each reads, all six stay barriers: loose ones took 392 us for 388 with sixteen;
//   inputs      with one sequence every CTA normalises and quantises the row itself. With more, one CTA per row does and leaves
//               the codes and a flag for all: reading b f32 rows in 148 places costs more than the extra step. The
//               residual stream stays in the registers of the CTA that needs it;
//   attention   teams of 4, 8 or 16 warps take slices of one sequence's and KV head's positions; a warp takes eight
//               positions at a time, a lane four dimensions, and the first keys and values are in registers before
//               the barrier in front. Slices are added up by one CTA or warp per head.
//
// Polling the values instead of a count (64-bit words with a number, or a flag per CTA): with 148 CTAs polling the lines that others write
// a step took 1.5 times as long.
//
// Measured, a whole step with head and argmax, a kernel per operation -> this: one sequence at 2000 positions, 30 layers of 2560,
// vocabulary 128256 1309 -> 787 us (of it 110 the head); sixteen sequences at 400 positions, 8 layers, vocabulary 32000 547 -> 370 us. At other widths,
// 512 to 8192, with 1 to 16 sequences at 100 and 2000 positions, 1.14 to 2.8 times as fast as a kernel per operation, rings of two stages included.
#include "lbk_gemv_core.cuh"

#include <exception>
#include <memory>
#include <new>

namespace lbk {

using namespace gemv;

namespace {

constexpr int kHead = 128;          // head size
constexpr int kGroup = 4;           // query heads per KV head at most
constexpr int kPhases = 4;          // q/k/v, o, gate/up, down
constexpr int kMaxRing = 8;
constexpr int kPositions = 8;       // positions a warp takes at a time
constexpr int kRecord = kHead + 4;  // floats of a slice's or warp's partial result: 128 sums, maximum, weight, padding
constexpr int kMaxSlices = 32;      // a lane each when they are added up
constexpr uint32_t kPollLimit = 1u << 20;  // polls of a count before a wait gives up, about a second (lbk_step_set_wait_limit)

struct alignas(16) LayerInfo {
    const float *norm[4];  // input, attention sub-norm, post-attention, feed-forward sub-norm
    float wscale[8];       // q, k, v, o, gate, up, down
};
constexpr int kInfoWords = sizeof(LayerInfo) / 4;
struct alignas(128) StepLayer {
    CUtensorMap tmap[7];   // in the order of wscale
    LayerInfo info;
};

struct Phase {
    int n_mat, first, chunks, k, tiles;
    int tile_end[3], rows[3];
    float *out[3];         // [m][rows] of each matrix; gate/up: [m][rows] of relu(gate)^2 up in out[0]
};

struct StepParams {
    int layers, m, heads, kv_heads, cap, ring, list;  // list: stages of a layer a warp has at most
    int team_warps, slices, pos_stride;
    int region, acc_ints;       // bytes of the input / attention area, ints of the sums
    float eps, scaling;
    const StepLayer *table;
    const float *final_norm;
    const float *x;             // [m][hidden], the embedded tokens
    float *attn, *part;         // [m][heads][128]; [m][kv_heads][kGroup][slices][kRecord]
    float *out;
    const float *cos, *sin;
    const int32_t *pos;
    uint16_t *kcache, *vcache;
    size_t layer_stride;        // elements of a layer's cache
    uint8_t *q8;                // [m][row] codes in fragment order
    float *q8_scale;
    int32_t *q8_sum;
    // of all launches so far: meetings, rows of codes, layers; arrivals at meetings, rows of codes that are there; and the CTAs that have left this one
    uint32_t *number, *codes, *turn, *met, *q8_ready, *exit_count;
    uint64_t layout, *held;     // the sizes that the places lie by, in this launch and in the one before it on this buffer
    uint4 *places;              // all that Place stands for: behind the q/k/v rows, up to the codes
    uint32_t place_words;       // 16 bytes each
    int *err_word;
    uint32_t poll_limit;
    Phase ph[kPhases];
};

struct Layout {
    uint32_t bars, region, acc, part, run, cta, scale, sum, pos, flag, info, list, total;
};
__host__ __device__ inline Layout layout_of(int ring, int list, int region, int acc_ints) {
    Layout L;
    uint32_t o = kWarps * ring * kStageBytes;
    L.bars = o;   o += kWarps * kMaxRing * 8;
    L.run = o;    o += kWarps * kPhases * 16;
    L.cta = o;    o += kPhases * 8;
    L.part = o;   o += 3 * kWarps * 4;
    L.scale = o;  o += kMaxM * 4;
    L.sum = o;    o += kMaxM * 4;
    L.pos = o;    o += kMaxM * 4;
    L.flag = o;   o += 32;
    o = (o + 15u) & ~15u;
    L.info = o;   o += 2 * kInfoWords * 4;
    L.list = o;   o += kWarps * list * 8;
    o = (o + 127u) & ~127u;
    L.region = o; o += static_cast<uint32_t>(region);
    L.acc = o;    o += static_cast<uint32_t>(acc_ints) * 4;
    L.total = o;
    return L;
}
__host__ __device__ inline int row_stride(int chunks) { return chunks * kChunkCols + 64; }

__device__ __forceinline__ float bf16_value(uint32_t b) { return __uint_as_float(b << 16); }
__device__ __forceinline__ uint32_t to_bf16(float f) {  // nearest even, as the other cache writers
    uint32_t u = __float_as_uint(f);
    if ((u & 0x7fffffffu) > 0x7f800000u) return (u >> 16) | 0x40u;
    return (u + 0x7fffu + ((u >> 16) & 1u)) >> 16;
}
__device__ __forceinline__ float4 bf16x4(uint2 r) {
    return make_float4(bf16_value(r.x & 0xffffu), __uint_as_float(r.x & 0xffff0000u), bf16_value(r.y & 0xffffu), __uint_as_float(r.y & 0xffff0000u));
}
__device__ __forceinline__ float4 shfl_xor4(float4 v, int o) {
    return make_float4(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o), __shfl_xor_sync(0xffffffffu, v.z, o),
                       __shfl_xor_sync(0xffffffffu, v.w, o));
}
// How values go from one part to the next.
// LOOSE: behind a count that is not ordered after them. A float travels as its complement, so that a word of zeros means "not there yet" (the
// value it would stand for, a NaN that no arithmetic leaves, goes as another NaN), and every reader looks again until all words are there.
// There are two places for each value, taken in turn by the layers: whoever writes one clears the other. At that time all CTAs have met
// at this layer's barrier, behind their last look at the other, and they meet at the next before they look at it again.
// Otherwise as they are, behind a barrier.
template <bool LOOSE>
struct Place {
    float *at;
    ptrdiff_t other;  // floats from a place to the other
    static __device__ __forceinline__ uint32_t word(float v) {  // as it travels
        const uint32_t u = __float_as_uint(v);
        return !LOOSE ? u : u == ~0u ? ~0x7fffffffu : ~u;
    }
    static __device__ __forceinline__ float value(uint32_t u) { return __uint_as_float(LOOSE ? ~u : u); }
    static __device__ __forceinline__ uint4 words(float4 v) { return make_uint4(word(v.x), word(v.y), word(v.z), word(v.w)); }
    static __device__ __forceinline__ float4 values(uint4 u) { return make_float4(value(u.x), value(u.y), value(u.z), value(u.w)); }
    __device__ __forceinline__ void put(size_t i, float v) const {
        if constexpr (!LOOSE) {
            at[i] = v;
        } else {
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(at + i), "r"(word(v)) : "memory");
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(at + i + other), "r"(0u) : "memory");
        }
    }
    __device__ __forceinline__ void put2(size_t i, float2 v) const {
        if constexpr (!LOOSE) {
            *reinterpret_cast<float2 *>(at + i) = v;
        } else {
            asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(at + i), "r"(word(v.x)), "r"(word(v.y)) : "memory");
            asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %1};" ::"l"(at + i + other), "r"(0u) : "memory");
        }
    }
    __device__ __forceinline__ void put4(size_t i, float4 v) const {
        if constexpr (!LOOSE) {
            *reinterpret_cast<float4 *>(at + i) = v;
        } else {
            const uint4 u = words(v);
            asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(at + i), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w) : "memory");
            asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %1, %1, %1};" ::"l"(at + i + other), "r"(0u) : "memory");
        }
    }
    static __device__ __forceinline__ uint4 look4(const float *from) {
        if (!LOOSE) return __ldcg(reinterpret_cast<const uint4 *>(from));
        uint4 u;
        asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(from) : "memory");
        return u;
    }
    static __device__ __forceinline__ uint2 look2(const float *from) {
        if (!LOOSE) return __ldcg(reinterpret_cast<const uint2 *>(from));
        uint2 u;
        asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(u.x), "=r"(u.y) : "l"(from) : "memory");
        return u;
    }
};
__device__ __forceinline__ float4 ldcg4(const float *at) { return __ldcg(reinterpret_cast<const float4 *>(at)); }

// What a CTA carries through the step.
struct Cta {
    uint8_t *sm;
    Layout L;
    int tid, lane, warp;
    int *err_word;
    // a layer's norms and scales, copied here a layer ahead: two words of memory in a row are a trip to HBM each
    __device__ __forceinline__ const LayerInfo &info(int layer) const { return reinterpret_cast<const LayerInfo *>(sm + L.info)[layer & 1]; }
    __device__ __forceinline__ void fetch_info(const StepLayer *table, int layer) const {
        if (tid < kInfoWords) reinterpret_cast<uint32_t *>(sm + L.info)[(layer & 1) * kInfoWords + tid] = __ldg(reinterpret_cast<const uint32_t *>(&table[layer].info) + tid);
    }
    __device__ __forceinline__ volatile int *gave_up() const { return reinterpret_cast<volatile int *>(sm + L.flag); }
    // a wait has run out: the step is lost, later waits are skipped and the rings run empty
    __device__ __forceinline__ void give_up() const {
        *gave_up() = 1;
        atomicExch(err_word, 1);
    }
};

// Counts what this CTA wrote before its last barrier of threads; and waits for a count.
__device__ __forceinline__ void count_up(uint32_t *at) { asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(at) : "memory"); }
__device__ __forceinline__ void await(const Cta &c, const StepParams &p, const uint32_t *at, uint32_t want) {
    if (*c.gave_up()) return;
    uint32_t seen, polls = 0;
    for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(at) : "memory");
        if (static_cast<int>(seen - want) >= 0) return;
        if (++polls >= p.poll_limit) break;
        __nanosleep(40);  // polls slow the arrivals down
    }
    c.give_up();
}
// All threads' writes before arrive() are seen by all threads of the grid after the matching wait().
__device__ __forceinline__ void arrive(const Cta &c, const StepParams &p) {
    __syncthreads();
    if (c.tid == 0) count_up(p.met);
}
// The same behind a part that hands its values on by Place<LOOSE>. LOOSE: the count only says when it is worth looking, and is not held up until the
// values have reached L2.
template <bool LOOSE>
__device__ __forceinline__ void arrive_behind(const Cta &c, const StepParams &p) {
    if (!LOOSE) return arrive(c, p);
    __syncthreads();
    if (c.tid == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(p.met) : "memory");
}
__device__ __forceinline__ void wait(const Cta &c, const StepParams &p, uint32_t number) {
    if (c.tid == 0) await(c, p, p.met, number * gridDim.x);
    __syncthreads();
}

// What look4() or look2() got, once it is there.
template <bool LOOSE>
__device__ __forceinline__ float4 settle(const Cta &c, const StepParams &p, const float *from, uint4 u) {
    if (LOOSE)
        for (uint32_t polls = 0; !u.x || !u.y || !u.z || !u.w; u = Place<true>::look4(from))
            if (*c.gave_up() || ++polls >= p.poll_limit) {
                c.give_up();
                break;
            }
    return Place<LOOSE>::values(u);
}
template <bool LOOSE>
__device__ __forceinline__ float2 settle(const Cta &c, const StepParams &p, const float *from, uint2 u) {
    if (LOOSE)
        for (uint32_t polls = 0; !u.x || !u.y; u = Place<true>::look2(from))
            if (*c.gave_up() || ++polls >= p.poll_limit) {
                c.give_up();
                break;
            }
    return make_float2(Place<LOOSE>::value(u.x), Place<LOOSE>::value(u.y));
}

// r of a row whose squares sum to ss; the scale of its codes from that sum and max|y|
__device__ __forceinline__ float norm_factor(float ss, int k, float eps) { return 1.0f / sqrtf(ss / static_cast<float>(k) + eps); }
__device__ __forceinline__ float scale_of(float2 row, int k, float eps) {
    return __fdiv_rn(127.0f, fmaxf(row.y * norm_factor(row.x, k, eps), 1e-5f));  // quant.rs:105
}
// A row through the norm and the quantiser, by the whole CTA: v holds it in float4 tid + 512 j, w the norm's weights. With
// y = x w and r the norm's factor the codes are round(y r 127 / max|y r|) = round(y 127 / max|y|): r only enters the scale, so the sum
// of squares and the maximum are reduced together, and the codes do not wait for r, whose two divisions and root took 500 of the 1800
// cycles: returned are the sum and the maximum, from which one thread has the scale (scale_of) beside or behind the codes. (The norm and
// quantise kernels round (x r w) (127 / max|x r w|): the same but for a code that lies on a rounding boundary to within a few units in
// the last place, a row of 2560 in some hundreds.) Leaves the codes (fragment order, zeros up to kfill) at dst and their sum
// in shared memory (quant.rs:101-118, model.rs:267-272).
template <int NJ>
__device__ __forceinline__ float2 norm_quant_row(const Cta &c, float4 (&v)[NJ], const float4 (&w)[NJ], int k, int kfill, float eps, uint8_t *dst) {
    float *s_ss = reinterpret_cast<float *>(c.sm + c.L.part), *s_max = s_ss + kWarps;
    int *s_sum = reinterpret_cast<int *>(s_max + kWarps);
    if (c.tid == 0) *s_sum = 0;
    float ss = 0.0f, am = 0.0f;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
        v[j] = make_float4(v[j].x * w[j].x, v[j].y * w[j].y, v[j].z * w[j].z, v[j].w * w[j].w);
        am = fmaxf(am, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(am)));  // not negative, and never NaN (fmaxf drops it): bits order as values
    if (c.lane == 0) {
        s_ss[c.warp] = ss;
        s_max[c.warp] = am;
    }
    __syncthreads();
    ss = am = 0.0f;
#pragma unroll
    for (int i = 0; i < kWarps; i += 4) {
        const float4 f = *reinterpret_cast<const float4 *>(s_ss + i), g = *reinterpret_cast<const float4 *>(s_max + i);
        ss += (f.x + f.y) + (f.z + f.w);
        am = fmaxf(am, fmaxf(fmaxf(g.x, g.y), fmaxf(g.z, g.w)));
    }
    float mult = __fdiv_rn(127.0f, am);  // of y, unless max|y r| < 1e-5 or no number: an estimate of it tells, at half the bound or closer the value itself
    if (!(am * rsqrtf(__fdividef(ss, static_cast<float>(k)) + eps) >= 2e-5f)) {
        const float r = norm_factor(ss, k, eps);
        if (!(am * r >= 1e-5f)) mult = r * scale_of(make_float2(ss, am), k, eps);
    }
    int total = 0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int i = (c.tid + j * kThreads) * 4;
        if (i < kfill) {
            const int q0 = quant_one(v[j].x, mult), q1 = quant_one(v[j].y, mult), q2 = quant_one(v[j].z, mult), q3 = quant_one(v[j].w, mult);
            total += q0 + q1 + q2 + q3;
            *reinterpret_cast<uint32_t *>(dst + xq_pos(i)) = pack4(q0, q1, q2, q3);
        }
    }
    total = __reduce_add_sync(0xffffffffu, total);
    if (c.lane == 0) atomicAdd(s_sum, total);
    return make_float2(ss, am);
}

// This thread's part of row `row` of what the part in front left into v, added to the residual row x where `add` says so. The embedded tokens
// come as they are, everything else as Place<LOOSE> hands it on.
template <bool LOOSE, int NJ, int NX>
__device__ __forceinline__ void get_row(const Cta &c, const StepParams &p, int row, int k, const float *from, bool add, float4 (&x)[NX], float4 (&v)[NJ]) {
    const float *src = from + static_cast<size_t>(row) * k;
    const int n = k >> 2;
    if (!LOOSE || from == p.x) {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int i = c.tid + j * kThreads;
            v[j] = i < n ? ldcg4(src + i * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        uint4 u[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int i = c.tid + j * kThreads;
            u[j] = i < n ? Place<LOOSE>::look4(src + i * 4) : Place<LOOSE>::words(make_float4(0.f, 0.f, 0.f, 0.f));
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) v[j] = settle<LOOSE>(c, p, src + (c.tid + j * kThreads) * 4, u[j]);
    }
    if (add) {
#pragma unroll
        for (int j = 0; j < NX; ++j) x[j] = v[j] = make_float4(v[j].x + x[j].x, v[j].y + x[j].y, v[j].z + x[j].z, v[j].w + x[j].w);
    }
}

__device__ __forceinline__ int row_cta(int row) { return static_cast<int>(gridDim.x) - 1 - row; }

// The weight stream of a warp: a ring of stages, refilled through all phases of all layers. A layer's stages are listed in shared
// memory once (matrix and first row, first byte): worked out at each refill they cost about 1000 cycles.
struct Stream {
    uint32_t data, bars;
    const uint8_t *ptr;
    const int2 *list;
    int depth, each;  // stages in the ring, stages of a layer
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    int layer = 0, next = 0;  // lane 0: the next stage to fetch
    __device__ __forceinline__ void issue(const StepParams &p, int slot, uint64_t policy) {
        if (next == each) {
            next = 0;
            ++layer;
        }
        if (each == 0 || layer >= p.layers) return;
        const int2 e = list[next++];
        ptx::mbar_arrive_expect_tx(bars + slot * 8, kStageBytes);
        ptx::tma_load_2d_hint(data + slot * kStageBytes, &p.table[layer].tmap[e.x & 7], bars + slot * 8, e.y, e.x >> 3, policy);
    }
};

// From the barrier in front (the number-th) to codes, scales and sums of all rows in shared memory (SHARED: the last of `codes` rows so far).
template <int NJ, int NX, bool SHARED>
__device__ __forceinline__ float2 input_phase(const Cta &c, const StepParams &p, int phase, const float *from, uint32_t number, uint32_t codes, const float *w, float4 (&x)[NX]) {
    const Phase &ph = p.ph[phase];
    const int k = ph.k, kfill = ph.chunks * kChunkCols, stride = row_stride(ph.chunks);
    uint8_t *s_xq = c.sm + c.L.region;
    float *s_scale = reinterpret_cast<float *>(c.sm + c.L.scale);
    int *s_sum = reinterpret_cast<int *>(c.sm + c.L.sum);
    const int *s_codes = reinterpret_cast<const int *>(c.sm + c.L.part) + 2 * kWarps;
    const int row = SHARED ? row_cta(blockIdx.x) : 0;
    float2 sum_top = make_float2(0.f, 0.f);
    if (!SHARED || row < p.m) {
        float4 wv[NJ], v[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int i = c.tid + j * kThreads;
            wv[j] = i < (k >> 2) ? __ldg(reinterpret_cast<const float4 *>(w) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        wait(c, p, number);
        get_row<!SHARED>(c, p, row, k, from, (phase & 1) == 0, x, v);
        sum_top = norm_quant_row<NJ>(c, v, wv, k, kfill, p.eps, SHARED ? p.q8 + static_cast<size_t>(row) * stride : s_xq);
        if (SHARED && c.tid == kThreads - 1) p.q8_scale[row] = scale_of(sum_top, k, p.eps);  // beside the other warps' codes
        __syncthreads();
        if (c.tid == 0) {
            if (SHARED) {
                p.q8_sum[row] = *s_codes;
                count_up(p.q8_ready);
            } else {
                s_sum[0] = *s_codes;  // read behind the barrier after the products
            }
        }
    }
    if (SHARED) {
        if (c.tid == 0) await(c, p, p.q8_ready, codes);
        __syncthreads();
        const uint32_t dst = ptx::smem_u32(s_xq);
        for (int i = c.tid; i < p.m * (stride >> 4); i += kThreads) ptx::cp_async_16(dst + i * 16, p.q8 + static_cast<size_t>(i) * 16);
        ptx::cp_async_commit();
        if (c.tid < p.m) {
            s_scale[c.tid] = __ldcg(p.q8_scale + c.tid);
            s_sum[c.tid] = __ldcg(p.q8_sum + c.tid);
        }
        ptx::cp_async_wait<0>();
        __syncthreads();
    }
    return sum_top;
}

// ROW: one sequence, on the integer pipes (consume_stage_row)
template <int MT, bool ROW>
__device__ __forceinline__ void product_phase(const Cta &c, const StepParams &p, int phase, float2 row, const float *ws, const Place<ROW> &to, Stream &st, uint64_t policy) {
    const Phase &ph = p.ph[phase];
    const int g = c.lane >> 2, t = c.lane & 3, m = ROW ? 1 : p.m;
    const LaneOffsets off = lane_offsets(c.lane);
    const uint8_t *s_xq = c.sm + c.L.region;
    const int stride = row_stride(ph.chunks);
    int *s_acc = reinterpret_cast<int *>(c.sm + c.L.acc);
    const int *s_sum = reinterpret_cast<const int *>(c.sm + c.L.sum);
    const float *s_scale = reinterpret_cast<const float *>(c.sm + c.L.scale);
    const int4 run = reinterpret_cast<const int4 *>(c.sm + c.L.run)[c.warp * kPhases + phase];
    const int2 cta = reinterpret_cast<const int2 *>(c.sm + c.L.cta)[phase];
    const float *wscale = ws + ph.first;
    const uint8_t *xrow[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        int tok = mt * 8 + g;
        tok = tok < m ? tok : m - 1;  // lanes past the last row read it again; what they get is dropped
        xrow[mt] = s_xq + static_cast<size_t>(tok) * stride + t * 16;
    }
    int sums[2][4] = {};
    int acc[MT][2][4][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[mt][h][kk][j] = 0;
    int tile = run.x, chunk = run.y;
    for (int item = 0; item < run.z; ++item) {
        if (!ptx::mbar_wait(st.bars + st.s * 8, st.phase, kWaitLimit)) st.ok = false;
        bool free;
        if constexpr (ROW) {
            consume_stage_row(st.ptr + st.s * kStageBytes, off, xrow[0], static_cast<uint32_t>(chunk) * kChunkCols, sums);
            free = stage_read(sums);
        } else {
            consume_stage<MT>(st.ptr + st.s * kStageBytes, off, xrow, static_cast<uint32_t>(chunk) * kChunkCols, acc);
            free = stage_read<MT>(acc);
        }
        if (free && c.lane == 0) st.issue(p, st.s, policy);
        if (++st.s == st.depth) {
            st.s = 0;
            st.phase ^= 1;
        }
        const bool done = ++chunk == ph.chunks;
        if (done || item + 1 == run.z) {
            int *rec = s_acc + (tile - cta.x) * m * kTileRows;
            if constexpr (ROW) {
                const int lo = sum_row(sums[0]), hi = sum_row(sums[1]);
                if (t < 2) atomicAdd(rec + g + 8 * t, t ? hi : lo);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) sums[0][kk] = sums[1][kk] = 0;
            } else
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int tok = mt * 8 + 2 * t + (j & 1);
                    const int v = take_acc<MT>(acc, mt, j);
                    if (tok < m) atomicAdd(rec + tok * kTileRows + g + ((j & 2) ? 8 : 0), v);
                }
        }
        if (done) {
            chunk = 0;
            ++tile;
        }
    }
    // One sequence: its scale is worked out here, by the warps that have the fewest stages, and not by one thread in front of all; a step of 30 layers
    // of 2560 821 -> 800 us.
    const float row_scale = ROW && c.tid < cta.y * kTileRows ? scale_of(row, ph.k, p.eps) : 0.0f;
    __syncthreads();  // all sums are in
    // dot = sum - sum of codes (gemm.rs:306-308), times 1 / (activation scale * weight scale) (gemm.rs:141)
    auto scaled = [&](int dot, int tok, float w) { return __fmul_rn(__int2float_rn(dot - s_sum[tok]), __fdiv_rn(1.0f, __fmul_rn(ROW ? row_scale : s_scale[tok], w))); };
    if (phase == 2) {  // relu(gate)^2 * up of tiles that lie side by side
        for (int e = c.tid; e < (cta.y >> 1) * m * kTileRows; e += kThreads) {
            const int tl = e / (m * kTileRows), rest = e - tl * (m * kTileRows), tok = rest >> 4;
            int *gate = s_acc + 2 * tl * m * kTileRows + rest, *up = gate + m * kTileRows;
            const int row = ((cta.x >> 1) + tl) * kTileRows + (rest & 15);
            if (row < ph.rows[0]) {
                const float a = fmaxf(scaled(*gate, tok, wscale[0]), 0.f);
                to.put(static_cast<size_t>(tok) * ph.rows[0] + row, a * a * scaled(*up, tok, wscale[1]));
            }
            *gate = *up = 0;
        }
        return;
    }
    for (int e = c.tid; e < cta.y * m * kTileRows; e += kThreads) {
        const int tl = e / (m * kTileRows), rest = e - tl * (m * kTileRows), tok = rest >> 4;
        const int tile_id = cta.x + tl;
        int mat = 0;
        while (mat < ph.n_mat - 1 && tile_id >= ph.tile_end[mat]) ++mat;
        const int row = (tile_id - (mat ? ph.tile_end[mat - 1] : 0)) * kTileRows + (rest & 15);
        if (row < ph.rows[mat]) {
            const size_t at = static_cast<size_t>(tok) * ph.rows[mat] + row;
            const float v = scaled(s_acc[e], tok, wscale[mat]);
            if (phase == 0) ph.out[mat][at] = v;
            else to.put(at, v);
        }
        s_acc[e] = 0;
    }
}

// Adds up n partial results of one head in shared memory, `step` floats apart, a lane four dimensions.
__device__ __forceinline__ float4 merge_records(const float *from, int n, int step, int lane, float &gm, float &gs) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    const float mi = lane < n ? from[static_cast<size_t>(lane) * step + kHead] : -INFINITY;
    const float li = lane < n ? from[static_cast<size_t>(lane) * step + kHead + 1] : 0.0f;
    gm = warp_max(mi);
    const float f = mi == -INFINITY ? 0.0f : __expf(mi - gm);  // no positions: weighs nothing
    gs = f * li;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) gs += __shfl_xor_sync(0xffffffffu, gs, d);
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
        const float fi = __shfl_sync(0xffffffffu, f, i);
        const float4 a = *reinterpret_cast<const float4 *>(from + static_cast<size_t>(i) * step + lane * 4);
        o.x += fi * a.x; o.y += fi * a.y; o.z += fi * a.z; o.w += fi * a.w;
    }
    return o;
}

// Adds up the slices of every head of every sequence. Up to four slices: a warp per head, a lane four dimensions. More: a warp per eight
// dimensions of a head, a lane a slice (16 such warps on one SM took 4900 cycles, spread over the SMs 1500). Either way all that a warp
// needs is asked for at once.
template <bool LOOSE>
__device__ __forceinline__ void merge_slices(const Cta &c, const StepParams &p, const float *part_at, const Place<LOOSE> &to) {
    using At = Place<LOOSE>;
    const int group = p.heads / p.kv_heads, heads = p.m * p.heads, S = p.slices;
    const bool per_warp = S <= 4;
    const int units = per_warp ? heads : heads * (kHead / 8);
    for (int unit = c.warp * gridDim.x + blockIdx.x; unit < units; unit += gridDim.x * kWarps) {
        const int u = per_warp ? unit : unit / (kHead / 8), part = per_warp ? 0 : unit % (kHead / 8);
        const int b = u / p.heads, h = u - b * p.heads, kh = h / group;
        const float *rec = part_at + (static_cast<size_t>(b * p.kv_heads + kh) * kGroup + (h - kh * group)) * S * kRecord;
        const size_t dst = static_cast<size_t>(u) * kHead;
        if (per_warp) {
            float2 ml[4];
            float4 v[4];
            uint2 ml_u[4];
            uint4 v_u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                ml_u[i] = i < S ? At::look2(rec + i * kRecord + kHead) : make_uint2(At::word(-INFINITY), At::word(0.f));
                v_u[i] = i < S ? At::look4(rec + i * kRecord + c.lane * 4) : At::words(make_float4(0.f, 0.f, 0.f, 0.f));
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                ml[i] = settle<LOOSE>(c, p, rec + i * kRecord + kHead, ml_u[i]);
                v[i] = settle<LOOSE>(c, p, rec + i * kRecord + c.lane * 4, v_u[i]);
            }
            const float gm = fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x));
            float gs = 0.0f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float f = ml[i].x == -INFINITY ? 0.0f : __expf(ml[i].x - gm);
                gs += f * ml[i].y;
                o.x += f * v[i].x; o.y += f * v[i].y; o.z += f * v[i].z; o.w += f * v[i].w;
            }
            const float inv = 1.0f / gs;
            to.put4(dst + c.lane * 4, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
        } else {
            const float *r = rec + c.lane * kRecord;
            const bool in = c.lane < S;
            const uint4 none = At::words(make_float4(0.f, 0.f, 0.f, 0.f));
            const uint2 ml_u = in ? At::look2(r + kHead) : make_uint2(At::word(-INFINITY), At::word(0.f));
            const uint4 a_u = in ? At::look4(r + part * 8) : none, e_u = in ? At::look4(r + part * 8 + 4) : none;
            const float2 ml = settle<LOOSE>(c, p, r + kHead, ml_u);
            const float4 a = settle<LOOSE>(c, p, r + part * 8, a_u), e = settle<LOOSE>(c, p, r + part * 8 + 4, e_u);
            const float gm = warp_max(ml.x), f = ml.x == -INFINITY ? 0.0f : __expf(ml.x - gm);
            float d[9] = {f * a.x, f * a.y, f * a.z, f * a.w, f * e.x, f * e.y, f * e.z, f * e.w, f * ml.y};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < 9; ++i) d[i] += __shfl_xor_sync(0xffffffffu, d[i], o);
            const float inv = 1.0f / d[8];
            if (c.lane == 0) to.put4(dst + part * 8, make_float4(d[0] * inv, d[1] * inv, d[2] * inv, d[3] * inv));
            if (c.lane == 1) to.put4(dst + part * 8 + 4, make_float4(d[4] * inv, d[5] * inv, d[6] * inv, d[7] * inv));
        }
    }
}

// Asks for the keys and values that this CTA takes in `layer`'s attention to come to L2, a layer ahead: asked for behind the q/k/v products they
// queued behind the weights of the next projections, which every SM fetches at that time, and the slowest slice was twice the usual one. 30 layers of 2560
// at 2000 positions 799 -> 787 us a step, 16 sequences at 400, eight layers 385 -> 378 (with the step's last kernel as it was then).
__device__ __forceinline__ void call_cache(const Cta &c, const StepParams &p, int layer) {
    const int TW = p.team_warps, teams = kWarps / TW, team = c.warp / TW, units = p.m * p.kv_heads * p.slices;
    if (c.tid - team * TW * 32 != 0 || p.layer_stride % 8) return;  // a bulk prefetch starts on 16 bytes; the loads themselves need 8
    const int *s_pos = reinterpret_cast<const int *>(c.sm + c.L.pos);
    for (int unit = blockIdx.x * teams + team; unit < units; unit += gridDim.x * teams) {
        const int pair = unit / p.slices, slice = unit - pair * p.slices, b = pair / p.kv_heads, kh = pair - b * p.kv_heads, pos = s_pos[b];
        const int per = (pos + p.slices) / p.slices, p0 = slice * per, p1 = min(min(pos, p.cap), p0 + per);  // rows of earlier tokens
        if (p1 <= p0) continue;
        const size_t at = static_cast<size_t>(layer) * p.layer_stride + ((static_cast<size_t>(b) * p.kv_heads + kh) * p.cap + p0) * kHead;
        const uint32_t bytes = static_cast<uint32_t>(p1 - p0) * kHead * 2;
        ptx::prefetch_l2(p.kcache + at, bytes);
        ptx::prefetch_l2(p.vcache + at, bytes);
    }
}

// Attention of the step's tokens over the cache (model.rs:334-357), f32 on bf16 keys and values.
template <bool LOOSE>
__device__ __forceinline__ void attention_phase(const Cta &c, const StepParams &p, int layer, uint32_t number, const Place<LOOSE> &attn, const Place<LOOSE> &part) {
    const int TW = p.team_warps, teams = kWarps / TW, team = c.warp / TW, wt = c.warp % TW, ttid = c.tid - team * TW * 32;
    const int group = p.heads / p.kv_heads, units = p.m * p.kv_heads * p.slices, bar = 1 + team, tthreads = TW * 32;
    const int *s_pos = reinterpret_cast<const int *>(c.sm + c.L.pos);
    float *s_rec = reinterpret_cast<float *>(c.sm + c.L.region) + static_cast<size_t>(team) * TW * kGroup * kRecord;
    bool waited = false;
    for (int unit = blockIdx.x * teams + team; unit < units || !waited; unit += gridDim.x * teams) {
        const bool have = unit < units;  // the barrier is for all warps
        const int pair = have ? unit / p.slices : 0, slice = have ? unit - pair * p.slices : 0;
        const int b = pair / p.kv_heads, kh = pair - b * p.kv_heads, pos = s_pos[b], total = pos + 1;
        const bool valid = have && pos >= 0 && pos < p.cap;  // checked here: a replay past the end must not touch other rows
        const int per = (total + p.slices - 1) / p.slices;
        const int p0 = slice * per, p1 = valid ? min(total, p0 + per) : 0;
        const size_t slab = static_cast<size_t>(layer) * p.layer_stride + (static_cast<size_t>(b) * p.kv_heads + kh) * p.cap * kHead + c.lane * 4;
        uint16_t *kb = p.kcache + slab, *vb = p.vcache + slab;
        uint2 kr[kPositions], vr[kPositions];
        auto fetch = [&](int pc) {  // rows of earlier tokens
#pragma unroll
            for (int j = 0; j < kPositions; ++j) {
                const int at = pc + j;
                const bool in = at < p1 && at != pos;
                kr[j] = in ? *reinterpret_cast<const uint2 *>(kb + static_cast<size_t>(at) * kHead) : make_uint2(0u, 0u);
                vr[j] = in ? *reinterpret_cast<const uint2 *>(vb + static_cast<size_t>(at) * kHead) : make_uint2(0u, 0u);
            }
        };
        int pc = p0 + wt * kPositions;
        fetch(pc);
        float4 cs = make_float4(0.f, 0.f, 0.f, 0.f), sn = cs;
        if (valid) {
            cs = __ldg(reinterpret_cast<const float4 *>(p.cos + static_cast<size_t>(pos) * kHead) + c.lane);
            sn = __ldg(reinterpret_cast<const float4 *>(p.sin + static_cast<size_t>(pos) * kHead) + c.lane);
        }
        if (!waited) {
            wait(c, p, number);  // q, k and v of this layer are there
            waited = true;
        }
        if (!valid) {
            if (have && ttid == 0) atomicExch(p.err_word, 7);
            if (LOOSE && have && wt < group) {  // whoever reads on waits for something
                if (p.slices == 1) attn.put4((static_cast<size_t>(b) * p.heads + kh * group + wt) * kHead + c.lane * 4, make_float4(0.f, 0.f, 0.f, 0.f));
                else {
                    const size_t dst = ((static_cast<size_t>(pair) * kGroup + wt) * p.slices + slice) * kRecord;
                    part.put4(dst + c.lane * 4, make_float4(0.f, 0.f, 0.f, 0.f));
                    if (c.lane == 0) part.put2(dst + kHead, make_float2(-INFINITY, 0.f));
                }
            }
            continue;
        }
        // x * cos + rotate_half(x) * sin (model.rs:298-302); lane and lane ^ 16 hold the two halves
        auto turn = [&](float4 x) {
            float4 o = shfl_xor4(x, 16);
            if (c.lane < 16) o = make_float4(-o.x, -o.y, -o.z, -o.w);
            return make_float4(x.x * cs.x + o.x * sn.x, x.y * cs.y + o.y * sn.y, x.z * cs.z + o.z * sn.z, x.w * cs.w + o.w * sn.w);
        };
        float4 q[kGroup], acc[kGroup];
#pragma unroll
        for (int h = 0; h < kGroup; ++h)
            q[h] = ldcg4(p.ph[0].out[0] + (static_cast<size_t>(b) * p.heads + kh * group + (h < group ? h : 0)) * kHead + c.lane * 4);
        const bool owner = pos >= p0 && pos < p1 && (pos - p0) / kPositions % TW == wt;  // the new token ends this warp's positions
        const size_t new_at = (static_cast<size_t>(b) * p.kv_heads + kh) * kHead + c.lane * 4;
        const float4 k_new = owner ? ldcg4(p.ph[0].out[1] + new_at) : cs, v_new = owner ? ldcg4(p.ph[0].out[2] + new_at) : cs;
#pragma unroll
        for (int h = 0; h < kGroup; ++h) {
            const float4 v = turn(q[h]);
            q[h] = make_float4(v.x * p.scaling, v.y * p.scaling, v.z * p.scaling, v.w * p.scaling);
            acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        uint2 kw = make_uint2(0u, 0u), vw = kw;  // its row: rounded as the cache holds it, and appended
        if (owner) {
            const float4 kn = turn(k_new);
            kw = make_uint2(to_bf16(kn.x) | to_bf16(kn.y) << 16, to_bf16(kn.z) | to_bf16(kn.w) << 16);
            vw = make_uint2(to_bf16(v_new.x) | to_bf16(v_new.y) << 16, to_bf16(v_new.z) | to_bf16(v_new.w) << 16);
            *reinterpret_cast<uint2 *>(kb + static_cast<size_t>(pos) * kHead) = kw;
            *reinterpret_cast<uint2 *>(vb + static_cast<size_t>(pos) * kHead) = vw;
        }
        float mx = -INFINITY, sum = 0.0f;  // of head lane / 8
        for (; pc < p1; pc += TW * kPositions) {
#pragma unroll
            for (int j = 0; j < kPositions; ++j)
                if (pc + j == pos) {
                    kr[j] = kw;
                    vr[j] = vw;
                }
            // 32 dot products, each spread over the warp: folding halves leaves lane l with head l / 8, position l % 8
            float d[kGroup * kPositions];
#pragma unroll
            for (int j = 0; j < kPositions; ++j) {
                const float4 k4 = bf16x4(kr[j]);
#pragma unroll
                for (int h = 0; h < kGroup; ++h) d[h * kPositions + j] = q[h].x * k4.x + q[h].y * k4.y + q[h].z * k4.z + q[h].w * k4.w;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const bool up = (c.lane & o) != 0;
#pragma unroll
                for (int i = 0; i < o; ++i) {
                    const float give = up ? d[i] : d[i + o], keep = up ? d[i + o] : d[i];
                    d[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
            const bool in = pc + (c.lane & 7) < p1;
            const float sc = in ? d[0] : -INFINITY;
            float nm = sc;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) nm = fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, o));
            nm = fmaxf(nm, mx);
            const float corr = __expf(mx - nm), wgt = in ? __expf(sc - nm) : 0.0f;
            float ws = wgt;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
            sum = sum * corr + ws;
            mx = nm;
#pragma unroll
            for (int h = 0; h < kGroup; ++h) {
                const float f = __shfl_sync(0xffffffffu, corr, h * 8);
                acc[h].x *= f; acc[h].y *= f; acc[h].z *= f; acc[h].w *= f;
            }
#pragma unroll
            for (int j = 0; j < kPositions; ++j) {
                const float4 v4 = bf16x4(vr[j]);
#pragma unroll
                for (int h = 0; h < kGroup; ++h) {
                    const float f = __shfl_sync(0xffffffffu, wgt, h * 8 + j);
                    acc[h].x += f * v4.x; acc[h].y += f * v4.y; acc[h].z += f * v4.z; acc[h].w += f * v4.w;
                }
            }
            fetch(pc + TW * kPositions);
        }
        // the team's warps meet
        float *rec = s_rec + static_cast<size_t>(wt) * kGroup * kRecord;
#pragma unroll
        for (int h = 0; h < kGroup; ++h) *reinterpret_cast<float4 *>(rec + h * kRecord + c.lane * 4) = acc[h];
        if ((c.lane & 7) == 0) {
            rec[(c.lane >> 3) * kRecord + kHead] = mx;
            rec[(c.lane >> 3) * kRecord + kHead + 1] = sum;
        }
        ptx::named_barrier(bar, tthreads);
        if (wt < group) {  // a warp per head
            float gm, gs;
            const float4 o = merge_records(s_rec + wt * kRecord, TW, kGroup * kRecord, c.lane, gm, gs);
            if (p.slices == 1) {
                const float inv = 1.0f / gs;
                attn.put4((static_cast<size_t>(b) * p.heads + kh * group + wt) * kHead + c.lane * 4, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
            } else {
                const size_t dst = ((static_cast<size_t>(pair) * kGroup + wt) * p.slices + slice) * kRecord;
                part.put4(dst + c.lane * 4, o);
                if (c.lane == 0) part.put2(dst + kHead, make_float2(gm, gs));
            }
        }
        ptx::named_barrier(bar, tthreads);  // the records are free again
    }
}

// NH, NI: float4 a thread holds of a row of the hidden width and of the feed-forward width.
template <int MT, bool SHARED, int NH, int NI>
__global__ void __launch_bounds__(kThreads, 1) step_kernel(const __grid_constant__ StepParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = ptx::smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    Cta c;
    c.sm = smem_raw + (base - raw);
    c.L = layout_of(p.ring, p.list, p.region, p.acc_ints);
    c.err_word = p.err_word;
    c.tid = threadIdx.x;
    c.lane = c.tid & 31;
    c.warp = c.tid >> 5;
    if (c.lane < kPhases) {
        const Phase &ph = p.ph[c.lane];
        const int of = c.lane == 2 ? 2 : 1;  // gate and up tiles stay together
        const int t0 = static_cast<int>(static_cast<long long>(blockIdx.x) * (ph.tiles / of) / gridDim.x) * of;
        const int t1 = static_cast<int>(static_cast<long long>(blockIdx.x + 1) * (ph.tiles / of) / gridDim.x) * of;
        const int stages = (t1 - t0) * ph.chunks, s0 = stages * c.warp / kWarps, s1 = stages * (c.warp + 1) / kWarps;
        reinterpret_cast<int4 *>(c.sm + c.L.run)[c.warp * kPhases + c.lane] = make_int4(t0 + s0 / ph.chunks, s0 % ph.chunks, s1 - s0, 0);
        if (c.warp == 0) reinterpret_cast<int2 *>(c.sm + c.L.cta)[c.lane] = make_int2(t0, t1 - t0);
    }
    if (c.tid < 8) reinterpret_cast<int *>(c.sm + c.L.flag)[c.tid] = 0;
    if (c.tid < p.m) reinterpret_cast<int *>(c.sm + c.L.pos)[c.tid] = p.pos[c.tid * p.pos_stride];
    for (int i = c.tid; i < p.acc_ints; i += kThreads) reinterpret_cast<int *>(c.sm + c.L.acc)[i] = 0;
    c.fetch_info(p.table, 0);
    __syncwarp();
    Stream st;
    st.data = base + c.warp * p.ring * kStageBytes;
    st.ptr = c.sm + static_cast<size_t>(c.warp) * p.ring * kStageBytes;
    st.bars = base + c.L.bars + c.warp * (kMaxRing * 8);
    st.depth = p.ring;
    int2 *list = reinterpret_cast<int2 *>(c.sm + c.L.list) + c.warp * p.list;
    st.list = list;
    st.each = 0;
    for (int ph = 0; ph < kPhases; ++ph) {
        const Phase &f = p.ph[ph];
        const int4 run = reinterpret_cast<const int4 *>(c.sm + c.L.run)[c.warp * kPhases + ph];
        for (int i = c.lane; i < run.z; i += 32) {
            const int tile = run.x + (run.y + i) / f.chunks, chunk = (run.y + i) % f.chunks;
            int mat = 0, of = tile;
            if (ph == 2) {  // gate and up tiles in turn
                mat = tile & 1;
                of = tile >> 1;
            } else {
                while (mat < f.n_mat - 1 && tile >= f.tile_end[mat]) ++mat;
                if (mat) of -= f.tile_end[mat - 1];
            }
            list[st.each + i] = make_int2((of * kTileRows) << 3 | (f.first + mat), chunk * kChunkBytes);
        }
        st.each += run.z;
    }
    __syncwarp();
    const uint64_t policy = ptx::policy_evict_first();  // weights are read once per step
    if (c.lane == 0) {
        for (int i = 0; i < p.ring; ++i) ptx::mbar_init(st.bars + i * 8, 1);
        ptx::fence_barrier_init();
        for (int i = 0; i < p.ring; ++i) st.issue(p, i, policy);
    }
    __syncthreads();

    constexpr bool LOOSE = !SHARED;
    uint32_t number = *p.number, codes = *p.codes, turn = *p.turn;  // meetings, rows of codes and layers so far
    // A launch of other sizes has left its values where this one's places lie: they are cleared, by all, in front of the first barrier, behind which
    // the first place is written or looked at. (With several sequences values do not tell whether they are there.)
    if (LOOSE && *p.held != p.layout)
        for (uint32_t i = blockIdx.x * kThreads + c.tid; i < p.place_words; i += gridDim.x * kThreads) p.places[i] = make_uint4(0u, 0u, 0u, 0u);
    auto meet = [&] {
        arrive_behind<LOOSE>(c, p);
        ++number;
    };
    auto place = [&](float *two, size_t floats) {  // this layer's of the two
        const ptrdiff_t n = static_cast<ptrdiff_t>(floats);
        return LOOSE && (turn & 1) ? Place<LOOSE>{two + n, -n} : Place<LOOSE>{two, n};
    };
    float4 x[NH];  // the residual row: of the one sequence, or of the sequence that this CTA serves
#pragma unroll
    for (int j = 0; j < NH; ++j) x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float *from = p.x;
    call_cache(c, p, 0);
    // One copy of each part's code for all layers and projections: instructions that are fetched once a layer come from L2 otherwise.
#pragma unroll 1
    for (int l = 0; l < p.layers; ++l) {
        const LayerInfo &info = c.info(l);
        if (l + 1 < p.layers) c.fetch_info(p.table, l + 1);
#pragma unroll 1
        for (int ph = 0; ph < kPhases; ++ph) {
            if (SHARED) codes += p.m;
            const float2 row = input_phase<NI, NH, SHARED>(c, p, ph, from, number, codes, info.norm[ph], x);
            const Place<LOOSE> to = place(p.ph[ph].out[0], static_cast<size_t>(p.m) * p.ph[ph].rows[0]);
            product_phase<MT, !SHARED>(c, p, ph, row, info.wscale, to, st, policy);
            if (ph != 0) {
                meet();
                from = to.at;
                continue;
            }
            arrive(c, p);  // the one barrier of the layer: keys, values and queries go on as they are, and the places of the layer before are free
            ++number;
            const Place<LOOSE> attn = place(p.attn, static_cast<size_t>(p.m) * p.heads * kHead);
            const Place<LOOSE> part = place(p.part, static_cast<size_t>(p.m) * p.kv_heads * kGroup * p.slices * kRecord);
            attention_phase(c, p, l, number, attn, part);
            meet();
            if (p.slices > 1) {
                wait(c, p, number);
                merge_slices(c, p, part.at, attn);
                meet();
            }
            from = attn.at;
            if (l + 1 < p.layers) call_cache(c, p, l + 1);
        }
        ++turn;
    }
    wait(c, p, number);
    // the model's last norm, a CTA per row
    if (row_cta(blockIdx.x) < p.m) {
        const int k = p.ph[0].k, row = row_cta(blockIdx.x);
        float *s_ss = reinterpret_cast<float *>(c.sm + c.L.part);
        float4 v[NH];
        get_row<!SHARED>(c, p, row, k, from, true, x, v);
        float ss = 0.0f;
#pragma unroll
        for (int j = 0; j < NH; ++j) ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (c.lane == 0) s_ss[c.warp] = ss;
        __syncthreads();
        ss = 0.0f;
        for (int i = 0; i < kWarps; ++i) ss += s_ss[i];
        const float r = 1.0f / sqrtf(ss / static_cast<float>(k) + p.eps);
#pragma unroll
        for (int j = 0; j < NH; ++j) {
            const int i = c.tid + j * kThreads;
            if (i < (k >> 2)) {
                const float4 w = __ldg(reinterpret_cast<const float4 *>(p.final_norm) + i);
                reinterpret_cast<float4 *>(p.out + static_cast<size_t>(row) * k)[i] = make_float4(v[j].x * r * w.x, v[j].y * r * w.y, v[j].z * r * w.z, v[j].w * r * w.w);
            }
        }
    }
    if (!st.ok && c.lane == 0) atomicExch(p.err_word, 1);
    if (c.tid == 0 && atomicAdd(p.exit_count, 1u) == gridDim.x - 1) {  // all have taken the number: the next launch goes on from here
        *p.number = number;
        *p.codes = codes;
        *p.turn = turn;
        *p.held = p.layout;
        *p.exit_count = 0;
    }
}

using StepKernel = void (*)(StepParams);
// rows of a width that a CTA holds as so many float4 a thread, fill of the last chunk included
int float4s(size_t cols) {
    const size_t fill = (cols + kChunkCols - 1) / kChunkCols * kChunkCols, n = (fill + 4 * kThreads - 1) / (4 * kThreads);
    return n <= 2 ? 2 : n <= 4 ? 4 : n <= 8 ? 8 : 0;
}
template <int MT, bool SHARED>
StepKernel pick(int nh, int ni) {
    if (nh > ni) ni = nh;
    if (nh == 2) return ni == 2 ? step_kernel<MT, SHARED, 2, 2> : ni == 4 ? step_kernel<MT, SHARED, 2, 4> : step_kernel<MT, SHARED, 2, 8>;
    return ni <= 4 ? step_kernel<MT, SHARED, 4, 4> : step_kernel<MT, SHARED, 4, 8>;
}
StepKernel kernel_of(size_t b, int nh, int ni) { return b == 1 ? pick<1, false>(nh, ni) : b <= 8 ? pick<1, true>(nh, ni) : pick<2, true>(nh, ni); }

size_t round_up(size_t v) { return (v + 255) / 256 * 256; }

// Whether a stream may use every SM: one of a green context has a part of them, on which the grid cannot be resident as a whole.
bool stream_has_all(const Ctx *ctx, cudaStream_t st) {
    auto entry = [](const char *name) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? f : nullptr;
    };
    static const auto green_of = reinterpret_cast<CUresult (*)(CUstream, CUgreenCtx *)>(entry("cuStreamGetGreenCtx"));
    static const auto resource = reinterpret_cast<CUresult (*)(CUgreenCtx, CUdevResource *, CUdevResourceType)>(entry("cuGreenCtxGetDevResource"));
    CUgreenCtx green = nullptr;
    if (!green_of || !resource || green_of(st, &green) != CUDA_SUCCESS || !green) return true;
    CUdevResource r{};
    return resource(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS && r.sm.smCount >= static_cast<unsigned>(ctx->sm_count);
}

}  // namespace

struct Step {
    Ctx *ctx = nullptr;
    int device = 0;              // of its own: the step may be freed after the context
    size_t layers = 0, hidden = 0, inner = 0, heads = 0, kv_heads = 0;
    float eps = 0.0f;
    const float *final_norm = nullptr;
    StepLayer *table = nullptr;  // device
    bool served = false;
    uint32_t poll_limit = kPollLimit;
    int nh = 0, ni = 0;          // float4 a thread holds of a row of the hidden and of the feed-forward width
    ~Step() {
        if (table) cudaFree(table);
    }
    size_t rows(int ph, int mat) const { return ph == 0 ? (mat ? kv_heads : heads) * kHead : ph == 2 ? inner : hidden; }
    size_t cols(int ph) const { return ph == 1 ? heads * kHead : ph == 3 ? inner : hidden; }
    static int mats(int ph) { return ph == 0 ? 3 : ph == 2 ? 2 : 1; }

    // sizes, rings and teams for b sequences; pointers are left out
    bool plan(size_t b, size_t cap, StepParams &p) const {
        if (!served || b == 0 || b > static_cast<size_t>(kMaxM) || cap == 0) return false;
        p = StepParams{};
        p.layers = static_cast<int>(layers);
        p.m = static_cast<int>(b);
        p.heads = static_cast<int>(heads);
        p.kv_heads = static_cast<int>(kv_heads);
        p.cap = static_cast<int>(cap);
        p.eps = eps;
        p.scaling = 1.0f / sqrtf(static_cast<float>(kHead));
        int first = 0, chunks_max = 0, tiles_max = 0;
        for (int i = 0; i < kPhases; ++i) {
            Phase &f = p.ph[i];
            f.n_mat = mats(i);
            f.first = first;
            first += f.n_mat;
            f.k = static_cast<int>(cols(i));
            f.chunks = static_cast<int>((cols(i) + kChunkCols - 1) / kChunkCols);
            for (int j = 0; j < f.n_mat; ++j) {
                f.rows[j] = static_cast<int>(rows(i, j));
                f.tiles += (f.rows[j] + kTileRows - 1) / kTileRows;
                f.tile_end[j] = f.tiles;
            }
            chunks_max = f.chunks > chunks_max ? f.chunks : chunks_max;
            const int each = (f.tiles + ctx->sm_count - 1) / ctx->sm_count + 2;
            p.list += (each * f.chunks + kWarps - 1) / kWarps;
            tiles_max = each > tiles_max ? each : tiles_max;
        }
        const int records = kWarps * kGroup * kRecord * 4;
        p.region = p.m * row_stride(chunks_max);
        if (p.region < records) p.region = records;
        p.acc_ints = tiles_max * p.m * kTileRows;
        const size_t fixed = layout_of(0, p.list, p.region, p.acc_ints).total + 1024;
        if (fixed > ctx->smem_optin) return false;
        p.ring = static_cast<int>((ctx->smem_optin - fixed) / (kWarps * kStageBytes));
        if (p.ring > kMaxRing) p.ring = kMaxRing;
        if (p.ring < 2) return false;
        // Whole CTAs a slice while two or more CTAs are there for each head of each sequence, smaller teams beyond; no slice
        // shorter than 64 positions of a full cache.
        const int pairs = p.m * p.kv_heads, sms = ctx->sm_count;
        p.team_warps = 2 * pairs <= sms ? 16 : pairs <= sms ? 8 : 4;
        const int teams = kWarps / p.team_warps * sms;
        p.slices = teams / pairs > 1 ? teams / pairs : 1;
        const int most = static_cast<int>((cap + 63) / 64);
        if (p.slices > most) p.slices = most;
        if (p.slices > kMaxSlices) p.slices = kMaxSlices;
        return true;
    }
    // places in the work buffer, which has to start as zeros
    size_t carve(StepParams &p, uint8_t *base) const {
        size_t at = 0;
        auto take = [&](size_t bytes) {
            uint8_t *r = base + at;
            at += round_up(bytes);
            return r;
        };
        auto floats = [&](size_t n) { return reinterpret_cast<float *>(take(n * sizeof(float))); };
        const size_t b = p.m;
        p.number = reinterpret_cast<uint32_t *>(take(24));
        p.codes = p.number + 1;
        p.exit_count = p.number + 2;
        p.turn = p.number + 3;
        p.held = reinterpret_cast<uint64_t *>(p.number + 4);
        p.met = reinterpret_cast<uint32_t *>(take(4));
        p.q8_ready = reinterpret_cast<uint32_t *>(take(4));
        for (int i = 0; i < kPhases; ++i)
            for (int j = 0; j < (i == 2 ? 1 : p.ph[i].n_mat); ++j) p.ph[i].out[j] = floats((i ? 2 : 1) * b * p.ph[i].rows[j]);
        p.attn = floats(2 * b * heads * kHead);
        p.part = floats(2 * b * kv_heads * kGroup * p.slices * kRecord);
        p.places = reinterpret_cast<uint4 *>(p.ph[1].out[0]);
        p.place_words = static_cast<uint32_t>((base + at - reinterpret_cast<uint8_t *>(p.places)) / 16);
        // every size that `take` saw so far, none of them 0: hidden and inner are multiples of 4 and at most 8192 and 16384, heads at most 64
        p.layout = static_cast<uint64_t>(b) | static_cast<uint64_t>(p.slices) << 8 | static_cast<uint64_t>(heads) << 16 | static_cast<uint64_t>(kv_heads) << 24 |
                   static_cast<uint64_t>(hidden) << 32 | static_cast<uint64_t>(inner) << 48;
        int chunks = 0;
        for (const Phase &f : p.ph) chunks = f.chunks > chunks ? f.chunks : chunks;
        p.q8 = take(b * row_stride(chunks));
        p.q8_scale = floats(b);
        p.q8_sum = reinterpret_cast<int32_t *>(take(b * 4));
        return at;
    }
};

}  // namespace lbk

using namespace lbk;

extern "C" {

int lbk_step_create(lbk_ctx *c, size_t layers, const lbk_weight *const *linears, const float *const *norms, const float *final_norm, size_t heads,
                    size_t kv_heads, float eps, lbk_step **out) {
    if (!c || !linears || !norms || !final_norm || !out || !layers) return fail(LBK_ERR_INVALID, "lbk_step_create: null argument");
    if (!heads || !kv_heads || heads % kv_heads) return fail(LBK_ERR_INVALID, "lbk_step_create: inconsistent head counts");
    Ctx *ctx = reinterpret_cast<Ctx *>(c);
    LBK_CUDA(cudaSetDevice(ctx->device));
    std::unique_ptr<Step> s(new (std::nothrow) Step());
    if (!s) return fail(LBK_ERR_NOMEM, "out of host memory");
    s->ctx = ctx;
    s->device = ctx->device;
    s->layers = layers;
    s->heads = heads;
    s->kv_heads = kv_heads;
    s->eps = eps;
    s->final_norm = final_norm;
    std::vector<StepLayer> table;
    try {
        table.resize(layers);
    } catch (const std::exception &) {  // no exception leaves a C entry
        return fail(LBK_ERR_NOMEM, "lbk_step_create: no host memory for %zu layers", layers);
    }
    uintptr_t bits = reinterpret_cast<uintptr_t>(final_norm);
    for (size_t l = 0; l < layers; ++l) {
        const Weight *w[7];
        for (int i = 0; i < 7; ++i) {
            w[i] = reinterpret_cast<const Weight *>(linears[l * 7 + i]);
            if (!w[i]) return fail(LBK_ERR_INVALID, "lbk_step_create: projection %d of layer %zu is null", i, l);
        }
        if (l == 0) {
            s->hidden = w[0]->cols;
            s->inner = w[4]->rows;
        }
        for (int i = 0; i < 7; ++i) {
            const int ph = i < 3 ? 0 : i == 3 ? 1 : i < 6 ? 2 : 3, mat = ph == 0 ? i : ph == 2 ? i - 4 : 0;
            if (w[i]->rows != s->rows(ph, mat) || w[i]->cols != s->cols(ph))
                return fail(LBK_ERR_SHAPE, "lbk_step_create: projection %d of layer %zu is %zu x %zu", i, l, w[i]->rows, w[i]->cols);
            table[l].tmap[i] = w[i]->tmap_gemv;
            table[l].info.wscale[i] = w[i]->scale;
        }
        for (int i = 0; i < 4; ++i) {
            if (!norms[l * 4 + i]) return fail(LBK_ERR_INVALID, "lbk_step_create: norm %d of layer %zu is null", i, l);
            table[l].info.norm[i] = norms[l * 4 + i];
            bits |= reinterpret_cast<uintptr_t>(norms[l * 4 + i]);
        }
    }
    const size_t a = heads * kHead;
    s->nh = float4s(s->hidden > a ? s->hidden : a);
    s->ni = float4s(s->inner);
    s->served = heads / kv_heads <= kGroup && s->hidden && s->inner && s->hidden % 4 == 0 && s->inner % 4 == 0 && (s->nh == 2 || s->nh == 4) && s->ni != 0 && (bits & 15) == 0;
    // One value for every model, once: the limit belongs to the kernel, and with a launch's own size set before each launch a model
    // lowered it under another thread's larger launch.
    if (s->served) {
        int cooperative = 0, resident = 0;
        LBK_CUDA(cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, ctx->device));
        s->served = cooperative != 0;
        for (const size_t b : {1, 8, 16}) {
            const StepKernel kernel = kernel_of(b, s->nh, s->ni);
            LBK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ctx->smem_optin)));
            LBK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kThreads, ctx->smem_optin));
            s->served = s->served && resident > 0;
        }
    }
    LBK_CUDA(cudaMalloc(&s->table, layers * sizeof(StepLayer)));
    LBK_CUDA(cudaMemcpy(s->table, table.data(), layers * sizeof(StepLayer), cudaMemcpyHostToDevice));
    *out = reinterpret_cast<lbk_step *>(s.release());
    return LBK_OK;
}

int lbk_step_free(lbk_step *h) {
    Step *s = reinterpret_cast<Step *>(h);
    if (!s) return LBK_OK;
    LBK_CUDA(cudaSetDevice(s->device));
    LBK_CUDA(cudaDeviceSynchronize());
    delete s;
    return LBK_OK;
}

int lbk_step_supported(const lbk_step *h, size_t b, size_t cap) {
    StepParams p;
    return h && reinterpret_cast<const Step *>(h)->plan(b, cap, p) ? 1 : 0;
}

int lbk_step_set_wait_limit(lbk_step *h, uint32_t polls) {
    if (!h) return fail(LBK_ERR_INVALID, "lbk_step_set_wait_limit: null argument");
    if (polls == 0) return fail(LBK_ERR_INVALID, "a wait limit of 0 polls would give up before looking");
    reinterpret_cast<Step *>(h)->poll_limit = polls;
    return LBK_OK;
}

int lbk_step_stream_supported(const lbk_step *h, void *stream) {
    const Step *s = reinterpret_cast<const Step *>(h);
    if (!s || cudaSetDevice(s->ctx->device) != cudaSuccess) return 0;
    return stream_has_all(s->ctx, static_cast<cudaStream_t>(stream)) ? 1 : 0;
}

size_t lbk_step_work_bytes(const lbk_step *h, size_t b, size_t cap) {
    StepParams p;
    const Step *s = reinterpret_cast<const Step *>(h);
    return s && s->plan(b, cap, p) ? s->carve(p, nullptr) : 0;
}

int lbk_step_run(const lbk_step *h, size_t b, size_t cap, const float *x_dev, uint16_t *kcache_dev, uint16_t *vcache_dev, size_t layer_elems,
                 const float *cos_dev, const float *sin_dev, const int32_t *pos_dev, int pos_stride, void *work_dev, float *out_dev, void *stream) {
    const Step *s = reinterpret_cast<const Step *>(h);
    if (!s || !x_dev || !kcache_dev || !vcache_dev || !cos_dev || !sin_dev || !pos_dev || !work_dev || !out_dev)
        return fail(LBK_ERR_INVALID, "lbk_step_run: null argument");
    StepParams p;
    if (!s->plan(b, cap, p)) return fail(LBK_ERR_UNSUPPORTED, "lbk_step_run: %zu sequences of this model are not served by one launch", b);
    if ((reinterpret_cast<uintptr_t>(x_dev) | reinterpret_cast<uintptr_t>(out_dev) | reinterpret_cast<uintptr_t>(work_dev) | reinterpret_cast<uintptr_t>(kcache_dev) |
         reinterpret_cast<uintptr_t>(vcache_dev) | reinterpret_cast<uintptr_t>(cos_dev) | reinterpret_cast<uintptr_t>(sin_dev)) & 15)
        return fail(LBK_ERR_UNSUPPORTED, "lbk_step_run needs 16-byte aligned buffers");
    if (layer_elems < b * s->kv_heads * cap * kHead || layer_elems % 4) return fail(LBK_ERR_SHAPE, "lbk_step_run: a layer's cache holds %zu elements", layer_elems);
    Ctx *ctx = s->ctx;
    LBK_CUDA(cudaSetDevice(ctx->device));
    if (!stream_has_all(ctx, static_cast<cudaStream_t>(stream)))
        return fail(LBK_ERR_UNSUPPORTED, "lbk_step_run: the stream has a part of the device's multiprocessors, the step needs them all");
    s->carve(p, static_cast<uint8_t *>(work_dev));
    p.table = s->table;
    p.final_norm = s->final_norm;
    p.x = x_dev;
    p.out = out_dev;
    p.cos = cos_dev;
    p.sin = sin_dev;
    p.pos = pos_dev;
    p.pos_stride = pos_stride;
    p.kcache = kcache_dev;
    p.vcache = vcache_dev;
    p.layer_stride = layer_elems;
    p.err_word = ctx->err_word;
    p.poll_limit = s->poll_limit;
    const StepKernel kernel = kernel_of(b, s->nh, s->ni);
    const size_t smem = layout_of(p.ring, p.list, p.region, p.acc_ints).total + 1024;
    void *args[] = {&p};
    // cooperative: the CTAs wait on one another, so all of them have to be resident
    LBK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(static_cast<unsigned>(ctx->sm_count)), dim3(kThreads), args, smem,
                                         static_cast<cudaStream_t>(stream)));
    ctx->launches++;
    return LBK_OK;
}

}  // extern "C"

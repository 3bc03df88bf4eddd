// Mixture of experts: routing and the few-token expert kernels.
//
// Router: z = W_router h (rows of a projection, f32), s = softmax(z) over all experts, the `top` largest are chosen
// (the lower index first among equals) and their s are the weights, not renormalised. Expert: down(relu2(up h)).
// A shared expert of the same form runs for every token, times the sigmoid of one gate logit per token.
//
//   moe_topk / moe_scan / moe_scatter   prompt passes: chosen experts and weights, expert offsets, the tokens' rows
//                    copied in expert order; the expert projections are then dense_gemm_kernel / dense_f32_kernel
//                    calls over the sorted rows (lbk_dense.cu), and the norm behind the layer gathers, weights and sums
//                    each token's rows (lbk_layernorm.cu).
//   moe_few_up_kernel, moe_few_down_kernel   up to 16 tokens, bf16. Bound: HBM, the chosen experts' weights once; the
//                    streaming loop is lbk_few.cuh's. The up kernel routes the tokens itself and folds the routing weight into
//                    the activation. In the down kernel a CTA owns output rows and walks the shared and all chosen
//                    experts' columns as one long K, so the result does not depend on any order of arrival. Eight tokens,
//                    6 of 64 experts of 2560 x 1408 each (about 35 chosen, 252 MB a projection): up 105 -> 46 us, down 147 ->
//                    47 us against kernels whose lanes loaded their MMA fragments from global memory (5.5 TB/s now). For the
//                    down kernel boxes of 18 rows count: with two boxes of 9 for the same rows it took 72 us, whatever
//                    was in flight; a box costs its warp a wait, a refill and a chain of four MMAs.
#include "lbk_dense.cuh"
#include "lbk_dense_dev.cuh"
#include "lbk_few.cuh"
#include "lbk_ptx.cuh"

namespace lbk {

namespace {

constexpr int kMaxTop = 32;
constexpr int kMaxExperts = 1024;

// One warp routes one token: softmax over E logits, then `top` rounds of "largest that is left". Lane l holds
// experts l, l + 32, ... Calls put(k, expert, weight) in every lane.
template <int R, typename F>
__device__ __forceinline__ void route_token(const float *z, int E, int top, int lane, F put) {
    float v[R];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int e = lane + 32 * i;
        v[i] = e < E ? z[e] : -INFINITY;
        mx = fmaxf(mx, v[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int e = lane + 32 * i;
        v[i] = e < E ? expf(v[i] - mx) : -1.0f;
        if (e < E) sum += v[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    for (int k = 0; k < top; ++k) {
        float bv = -1.0f;
        int be = 1 << 30;
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (v[i] > bv) {
                bv = v[i];
                be = lane + 32 * i;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oe = __shfl_xor_sync(0xffffffffu, be, o);
            if (ov > bv || (ov == bv && oe < be)) {
                bv = ov;
                be = oe;
            }
        }
        if (be >= E) be = 0, bv = 0.0f;  // every logit is a NaN: any expert, weight zero
        put(k, be, bv / sum);
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (lane + 32 * i == be) v[i] = -2.0f;
    }
}

// ---- prompt passes --------------------------------------------------------------------------------
template <int R>
__global__ void __launch_bounds__(128) moe_topk_kernel(const float *z, long ldz, int n, int E, int top, int *ids, float *weight, int *counts) {
    ptx::pdl_trigger();
    ptx::pdl_wait();
    const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= n) return;
    route_token<R>(z + static_cast<size_t>(t) * ldz, E, top, lane, [&](int k, int e, float w) {
        if (lane == 0) {
            ids[t * top + k] = e;
            weight[t * top + k] = w;
            atomicAdd(counts + e, 1);
        }
    });
}

// offs = exclusive sums of counts; cursor starts there; counts go back to zero for the next pass
__global__ void __launch_bounds__(1024) moe_scan_kernel(int *counts, int *offs, int *cursor, int E) {
    ptx::pdl_trigger();
    ptx::pdl_wait();
    __shared__ int s[kMaxExperts];
    const int e = threadIdx.x;
    int c = e < E ? counts[e] : 0;
    s[e] = c;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int add = e >= o ? s[e - o] : 0;
        __syncthreads();
        s[e] += add;
        __syncthreads();
    }
    if (e < E) {
        offs[e] = cursor[e] = s[e] - c;
        counts[e] = 0;
        if (e == E - 1) offs[E] = s[e];
    }
}

// A block per token: its places in the sorted order, its row copied there (16-byte units).
__global__ void __launch_bounds__(128) moe_scatter_kernel(const int *ids, int top, int *cursor, int *place, int *token, const uint4 *x, long ldx16, int units,
                                                          uint4 *xs) {
    ptx::pdl_trigger();
    ptx::pdl_wait();
    __shared__ int s_place[kMaxTop];
    const int t = blockIdx.x;
    if (threadIdx.x < static_cast<unsigned>(top)) {
        const int p = atomicAdd(cursor + ids[t * top + threadIdx.x], 1);
        s_place[threadIdx.x] = p;
        place[t * top + threadIdx.x] = p;
        token[p] = t;
    }
    if (!xs) return;
    __syncthreads();
    for (int i = threadIdx.x; i < units; i += 128) {
        const uint4 v = x[static_cast<size_t>(t) * ldx16 + i];
        for (int k = 0; k < top; ++k) xs[static_cast<size_t>(s_place[k]) * units + i] = v;
    }
}

// ---- few tokens -------------------------------------------------------------------------------------
using few::kThreads;
using few::kTiles;
using few::kWarps;

struct FewMoeParams {
    alignas(64) CUtensorMap up;      // bytes [experts * ff][pitch * 2], box [16][128]
    alignas(64) CUtensorMap down;    // bytes [experts * width][pitch * 2], box [box_rows][128]
    alignas(64) CUtensorMap sdown;   // bytes [width][pitch * 2], box [box_rows][128]
    const uint16_t *n;
    long ldn;
    int m;
    const float *z;
    long ldz;
    int experts, top;
    size_t down_pitch, sdown_pitch;
    int up_chunks, down_chunks, sdown_chunks;  // of 64 columns
    int ff, width, ff_tiles, box_rows, boxes;  // down: a CTA's rows are `boxes` times box_rows
    uint16_t *h;
    const uint16_t *hs;
    float *y;
    int *act;       // [0]: number of chosen experts, then (expert, 16 slots packed as bytes: 4 ints) each
    int *err_word;
};
constexpr int kActInts = 5;

// The chosen experts' up projections: their tiles of 16 rows, one after the other, are dealt to the CTAs.
template <int NTL, int R>
__global__ void __launch_bounds__(kThreads, 1) moe_few_up_kernel(const __grid_constant__ FewMoeParams p) {
    extern __shared__ uint8_t moe_smem[];
    __shared__ int s_ids[LBK_GEMV_MAX_M][kMaxTop];
    __shared__ float s_wt[LBK_GEMV_MAX_M][kMaxTop];
    __shared__ unsigned s_mask[kMaxExperts];
    __shared__ short s_act[LBK_GEMV_MAX_M * kMaxTop];
    __shared__ int s_n;
    const uint32_t raw = ptx::smem_u32(moe_smem), base = (raw + 1023u) & ~1023u;
    uint8_t *sm = moe_smem + (base - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    few::Ring ring(sm, base, warp, 16);
    ptx::pdl_trigger();
    if (lane == 0) ring.init();
    for (int e = tid; e < p.experts; e += kThreads) s_mask[e] = 0u;
    __syncthreads();
    ptx::pdl_wait();
    if (warp < p.m)
        route_token<R>(p.z + static_cast<size_t>(warp) * p.ldz, p.experts, p.top, lane, [&](int k, int e, float w) {
            if (lane == 0) {
                s_ids[warp][k] = e;
                s_wt[warp][k] = w;
                atomicOr(&s_mask[e], 1u << warp);
            }
        });
    __syncthreads();
    if (warp == 0) {  // the chosen experts in ascending order
        int cnt = 0;
        for (int e0 = 0; e0 < p.experts; e0 += 32) {
            const bool on = e0 + lane < p.experts && s_mask[e0 + lane] != 0u;
            const unsigned bal = __ballot_sync(0xffffffffu, on);
            if (on) s_act[cnt + __popc(bal & ((1u << lane) - 1u))] = static_cast<short>(e0 + lane);
            cnt += __popc(bal);
        }
        if (lane == 0) s_n = cnt;
    }
    __syncthreads();
    const int n_act = s_n;
    auto slot_of = [&](int tk, int e) {  // which of token tk's choices expert e is, -1: none
        if (tk >= p.m || !((s_mask[e] >> tk) & 1u)) return -1;
        int k = 0;
        while (k < p.top - 1 && s_ids[tk][k] != e) ++k;
        return k;
    };
    const int units = n_act * p.ff_tiles, cta = static_cast<int>(blockIdx.x), ctas = static_cast<int>(gridDim.x);
    const int u0 = static_cast<int>(static_cast<long long>(units) * cta / ctas), u1 = static_cast<int>(static_cast<long long>(units) * (cta + 1) / ctas);
    const int total = few::chunks_of(p.up_chunks, warp) * (u1 - u0);
    struct Cursor {
        int q, k, c;
    } is{u0, 0, warp};
    auto load = [&](int slot) {
        const int u = is.q + is.k, a = u / p.ff_tiles;
        ring.fetch(slot, &p.up, is.c * 128, s_act[a] * p.ff + (u - a * p.ff_tiles) * 16);
        if (++is.k < min(kTiles, u1 - is.q)) return;
        is.k = 0;
        if ((is.c += kWarps) < p.up_chunks) return;
        is.c = warp;
        is.q += kTiles;
    };
    if (lane == 0)
        for (int i = 0; i < min(ring.depth, total); ++i) load(i);
    if (cta == 0) {  // the list for the down kernel
        if (tid == 0) p.act[0] = n_act;
        for (int a = tid; a < n_act; a += kThreads) {
            const int e = s_act[a];
            p.act[1 + a * kActInts] = e;
            for (int w = 0; w < 4; ++w) {
                unsigned word = 0;
                for (int i = 0; i < 4; ++i) word |= (static_cast<unsigned>(slot_of(w * 4 + i, e)) & 255u) << (8 * i);
                p.act[2 + a * kActInts + w] = static_cast<int>(word);
            }
        }
    }
    auto tokens = [&](few::Tokens<NTL> &x, int c) {
#pragma unroll
        for (int j = 0; j < NTL; ++j) {
            x.lo[j] = x.hi[j] = make_uint4(0u, 0u, 0u, 0u);
            if (j * 8 + g < p.m) {  // an expert meets every token; what it gives those that did not choose it is dropped
                const uint16_t *r = p.n + static_cast<size_t>(j * 8 + g) * p.ldn + c * 64 + t * 16;
                x.lo[j] = *reinterpret_cast<const uint4 *>(r);
                x.hi[j] = *reinterpret_cast<const uint4 *>(r + 8);
            }
        }
    };
    const few::Units place(lane);
    float *red = reinterpret_cast<float *>(sm + few::red_at());
    few::Tokens<NTL> x, x_next;
    if (warp < p.up_chunks) tokens(x_next, warp);
    int done = 0;
    for (int q = u0; q < u1; q += kTiles) {
        const int tiles = min(kTiles, u1 - q);
        float acc[kTiles][NTL][4];
        few::zero<NTL>(acc);
        for (int c = warp; c < p.up_chunks; c += kWarps) {
            x = x_next;
            tokens(x_next, c + kWarps < p.up_chunks ? c + kWarps : warp);
#pragma unroll
            for (int k = 0; k < kTiles; ++k)
                if (k < tiles) {
                    few::box_mma<NTL, 1>(ring.wait(), place, x, acc + k);
                    __syncwarp();
                    if (lane == 0 && done + ring.depth < total) load(ring.s);
                    ++done;
                    ring.next();
                }
        }
        if (q > u0) __syncthreads();  // the sums of the tiles before have been read
        few::leave<NTL>(red + warp * few::red_floats(NTL), lane, tiles, acc);
        __syncthreads();
        for (int o = tid; o < tiles * NTL * 128; o += kThreads) {
            const int k = o / (NTL * 128), f = o - k * (NTL * 128), tk = few::place_token(f);
            const int a = (q + k) / p.ff_tiles, r = (q + k - a * p.ff_tiles) * 16 + few::place_row(f);
            const int choice = slot_of(tk, s_act[a]);
            if (choice < 0 || r >= p.ff) continue;
            const float v = few::collect<NTL>(red, k, f);
            p.h[(static_cast<size_t>(tk) * p.top + choice) * p.down_pitch + r] = dense::f32_bf16(dense::relu2(v) * s_wt[tk][choice]);
        }
    }
    if (!ring.ok && lane == 0) atomicExch(p.err_word, 5);
}

// All down projections as one long K: the shared expert's columns (times its gate), then the chosen experts'.
template <int NTL, int MT>
__global__ void __launch_bounds__(kThreads, 1) moe_few_down_kernel(const __grid_constant__ FewMoeParams p) {
    extern __shared__ uint8_t moe_smem[];
    __shared__ short s_e[LBK_GEMV_MAX_M * kMaxTop];
    __shared__ signed char s_slot[LBK_GEMV_MAX_M * kMaxTop][16];
    const uint32_t raw = ptx::smem_u32(moe_smem), base = (raw + 1023u) & ~1023u;
    uint8_t *sm = moe_smem + (base - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    few::Ring ring(sm, base, warp, p.box_rows);
    constexpr int NB = kTiles / MT;  // boxes a warp carries at a time
    ptx::pdl_trigger();
    if (lane == 0) ring.init();
    ptx::pdl_wait();
    const int n_act = p.act[0];
    for (int a = tid; a < n_act; a += kThreads) {
        s_e[a] = static_cast<short>(p.act[1 + a * kActInts]);
        for (int w = 0; w < 4; ++w) *reinterpret_cast<int *>(&s_slot[a][4 * w]) = p.act[2 + a * kActInts + w];
    }
    __syncthreads();
    const int cs = p.hs ? p.sdown_chunks : 0, ce = p.down_chunks, chunks = cs + n_act * ce;
    const int total = few::chunks_of(chunks, warp) * p.boxes;
    const int row_base = static_cast<int>(blockIdx.x) * p.boxes * p.box_rows;
    // chunk c of the long K: the shared expert's, or chunk kk of the s-th chosen expert; steps of kWarps chunks
    struct Place {
        int c, s, kk;
    };
    auto place_at = [&](int c) { return Place{c, c < cs ? 0 : (c - cs) / ce, c < cs ? 0 : (c - cs) % ce}; };
    const Place start = place_at(warp);
    auto on = [&](Place &u) {
        const int before = u.c;
        u.c += kWarps;
        if (u.c >= chunks) {
            u = start;
            return true;
        }
        if (u.c >= cs) u.kk += before < cs ? u.c - cs : kWarps;
        while (u.kk >= ce) {
            u.kk -= ce;
            ++u.s;
        }
        return false;
    };
    Place is = start;
    int is_q = 0, is_k = 0;
    auto load = [&](int slot) {
        const int row = row_base + (is_q + is_k) * p.box_rows;
        if (is.c < cs) ring.fetch(slot, &p.sdown, is.c * 128, row);
        else ring.fetch(slot, &p.down, is.kk * 128, s_e[is.s] * p.width + row);
        if (++is_k < min(NB, p.boxes - is_q)) return;
        is_k = 0;
        if (on(is)) is_q += NB;
    };
    if (lane == 0)
        for (int i = 0; i < min(ring.depth, total); ++i) load(i);
    auto tokens = [&](few::Tokens<NTL> &x, const Place &u) {
        const int kk = u.c < cs ? u.c : u.kk;
#pragma unroll
        for (int j = 0; j < NTL; ++j) {
            const int tk = j * 8 + g;
            x.lo[j] = x.hi[j] = make_uint4(0u, 0u, 0u, 0u);
            const uint16_t *r = nullptr;
            if (u.c < cs) {
                if (tk < p.m) r = p.hs + static_cast<size_t>(tk) * p.sdown_pitch;
            } else {
                const int choice = s_slot[u.s][tk];
                if (choice >= 0) r = p.h + (static_cast<size_t>(tk) * p.top + choice) * p.down_pitch;
            }
            if (r) {
                x.lo[j] = *reinterpret_cast<const uint4 *>(r + kk * 64 + t * 16);
                x.hi[j] = *reinterpret_cast<const uint4 *>(r + kk * 64 + t * 16 + 8);
            }
        }
    };
    float gate[NTL][2];
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int tk = j * 8 + 2 * t + i;
            gate[j][i] = p.hs && tk < p.m ? dense::sigmoid(p.z[static_cast<size_t>(tk) * p.ldz + p.experts]) : 0.0f;
        }
    const few::Units place(lane);
    float *red = reinterpret_cast<float *>(sm + few::red_at());
    few::Tokens<NTL> x, x_next;
    Place ahead = start;
    if (warp < chunks) tokens(x_next, ahead);
    int done = 0;
    for (int q = 0; q < p.boxes; q += NB) {
        const int boxes = min(NB, p.boxes - q);
        float acc[kTiles][NTL][4];
        few::zero<NTL>(acc);
        auto shared_done = [&]() {  // what has been added up so far is the shared expert's
#pragma unroll
            for (int k = 0; k < kTiles; ++k)
#pragma unroll
                for (int j = 0; j < NTL; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[k][j][i] *= gate[j][i & 1];
        };
        for (int c = warp; c < chunks; c += kWarps) {
            x = x_next;
            on(ahead);
            tokens(x_next, ahead);
            if (c >= cs && c < cs + kWarps) shared_done();
#pragma unroll
            for (int k = 0; k < NB; ++k)
                if (k < boxes) {
                    few::box_mma<NTL, MT>(ring.wait(), place, x, acc + k * MT);
                    __syncwarp();
                    if (lane == 0 && done + ring.depth < total) load(ring.s);
                    ++done;
                    ring.next();
                }
        }
        if (cs + ((warp - cs) & (kWarps - 1)) >= chunks) shared_done();  // this warp has none of the experts' chunks
        if (q) __syncthreads();  // the sums of the boxes before have been read
        few::leave<NTL>(red + warp * few::red_floats(NTL), lane, boxes * MT, acc);
        __syncthreads();
        for (int o = tid; o < boxes * MT * NTL * 128; o += kThreads) {
            const int tile = o / (NTL * 128), f = o - tile * (NTL * 128), in_box = (tile % MT) * 16 + few::place_row(f), tk = few::place_token(f);
            const int r = row_base + (q + tile / MT) * p.box_rows + in_box;
            if (in_box < p.box_rows && r < p.width && tk < p.m) p.y[static_cast<size_t>(tk) * p.width + r] = few::collect<NTL>(red, tile, f);
        }
    }
    if (!ring.ok && lane == 0) atomicExch(p.err_word, 5);
}

using FewMoeKernel = void (*)(FewMoeParams);
FewMoeKernel few_up(bool two, bool wide) {
    return two ? (wide ? moe_few_up_kernel<2, 32> : moe_few_up_kernel<2, 8>) : (wide ? moe_few_up_kernel<1, 32> : moe_few_up_kernel<1, 8>);
}
FewMoeKernel few_down(bool two, int mt) {
    if (two) return mt == 1 ? moe_few_down_kernel<2, 1> : moe_few_down_kernel<2, 2>;
    return mt == 1 ? moe_few_down_kernel<1, 1> : moe_few_down_kernel<1, 2>;
}

int moe_init(Ctx *ctx) {
    for (const bool two : {false, true})
        for (FewMoeKernel k : {few_up(two, false), few_up(two, true), few_down(two, 1), few_down(two, 2)})
            LBK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, few::rest_at(2) + 1024));
    return LBK_OK;
}
const InitHook kInitMoe(moe_init);

int check_route(size_t experts, size_t top) {
    if (experts == 0 || top == 0 || top > experts) return fail(LBK_ERR_INVALID, "routing %zu of %zu experts", top, experts);
    if (experts > static_cast<size_t>(kMaxExperts) || top > static_cast<size_t>(kMaxTop))
        return fail(LBK_ERR_UNSUPPORTED, "routing: at most %d experts, %d of them per token", kMaxExperts, kMaxTop);
    return LBK_OK;
}

}  // namespace

size_t moe_route_ints(size_t n, size_t experts, size_t top) { return 4 * n * top + 2 * (experts + 1) + kMaxExperts; }

// The counts come first and have room for every possible number of experts: they are zero at rest, whatever
// layer (with whatever number of experts) uses the block.
void moe_route_carve(MoeRoute &r, int *base, size_t n, size_t experts, size_t top) {
    r.counts = base;
    r.offs = r.counts + kMaxExperts;
    r.cursor = r.offs + experts + 1;
    r.ids = r.cursor + experts + 1;
    r.place = r.ids + n * top;
    r.token = r.place + n * top;
    r.weight = reinterpret_cast<float *>(r.token + n * top);
}

int launch_moe_route(Ctx *ctx, const float *z, long ldz, size_t n, size_t experts, size_t top, const MoeRoute &r, const void *x, long ldx, void *xs,
                     cudaStream_t st) {
    LBK_TRY(check_route(experts, top));
    if (n == 0) return LBK_OK;
    const dim3 grid(static_cast<unsigned>((n + 3) / 4));
    const int E = static_cast<int>(experts), k = static_cast<int>(top);
    if (E <= 256) LBK_CUDA(launch_chained(moe_topk_kernel<8>, grid, dim3(128), 0, st, z, ldz, static_cast<int>(n), E, k, r.ids, r.weight, r.counts));
    else LBK_CUDA(launch_chained(moe_topk_kernel<32>, grid, dim3(128), 0, st, z, ldz, static_cast<int>(n), E, k, r.ids, r.weight, r.counts));
    LBK_CUDA(launch_chained(moe_scan_kernel, dim3(1), dim3(1024), 0, st, r.counts, r.offs, r.cursor, E));
    LBK_CUDA(launch_chained(moe_scatter_kernel, dim3(static_cast<unsigned>(n)), dim3(128), 0, st, r.ids, k, r.cursor, r.place, r.token,
                            static_cast<const uint4 *>(x), ldx / 8, static_cast<int>(ldx / 8), static_cast<uint4 *>(xs)));
    LBK_CUDA(cudaGetLastError());
    ctx->launches += 3;
    return LBK_OK;
}

int launch_moe_few(Ctx *ctx, const MoeFewCall &c, cudaStream_t st) {
    LBK_TRY(check_route(static_cast<size_t>(c.experts), static_cast<size_t>(c.top)));
    if (c.m == 0) return LBK_OK;
    if (c.m > LBK_GEMV_MAX_M) return fail(LBK_ERR_INVALID, "the few-token expert kernels take up to %d tokens", LBK_GEMV_MAX_M);
    FewMoeParams p{};
    p.n = c.n;
    p.ldn = c.ldn;
    p.m = static_cast<int>(c.m);
    p.z = c.z;
    p.ldz = c.ldz;
    p.experts = c.experts;
    p.top = c.top;
    p.down_pitch = c.down.pitch;
    p.up_chunks = static_cast<int>(c.up.pitch / 64);
    p.down_chunks = static_cast<int>(c.down.pitch / 64);
    p.ff = static_cast<int>(c.ff);
    p.width = static_cast<int>(c.width);
    p.ff_tiles = (p.ff + 15) / 16;
    p.h = c.h;
    p.y = c.y;
    p.act = c.act;
    p.err_word = ctx->err_word;
    const few::Deal deal = few::deal_rows(c.width, ctx->sm_count);
    p.box_rows = deal.box_rows;
    p.boxes = deal.boxes;
    LBK_TRY(encode_bytes_map(&p.up, c.up.w, c.up.pitch * 2, c.up.rows, c.up.pitch * 2, 128, 16));
    LBK_TRY(encode_bytes_map(&p.down, c.down.w, c.down.pitch * 2, c.down.rows, c.down.pitch * 2, 128, deal.box_rows));
    if (c.hs) {
        p.hs = c.hs;
        p.sdown_pitch = c.shared_down.pitch;
        p.sdown_chunks = static_cast<int>(c.shared_down.pitch / 64);
        LBK_TRY(encode_bytes_map(&p.sdown, c.shared_down.w, c.shared_down.pitch * 2, c.shared_down.rows, c.shared_down.pitch * 2, 128, deal.box_rows));
    }
    const size_t most = c.m * c.top < static_cast<size_t>(c.experts) ? c.m * c.top : static_cast<size_t>(c.experts);
    const size_t units = most * p.ff_tiles;
    const dim3 gu(static_cast<unsigned>(units < static_cast<size_t>(ctx->sm_count) ? units : ctx->sm_count));
    const bool two = c.m > 8;
    const size_t smem = static_cast<size_t>(few::rest_at(two ? 2 : 1)) + 1024;
    LBK_CUDA(launch_chained(few_up(two, c.experts > 256), gu, dim3(kThreads), smem, st, p));
    LBK_CUDA(launch_chained(few_down(two, deal.box_rows > 16 ? 2 : 1), dim3(static_cast<unsigned>(deal.ctas)), dim3(kThreads), smem, st, p));
    LBK_CUDA(cudaGetLastError());
    ctx->launches += 2;
    return LBK_OK;
}

size_t moe_few_act_ints(size_t m, size_t experts, size_t top) {
    const size_t most = m * top < experts ? m * top : experts;
    return 1 + most * kActInts;
}

}  // namespace lbk

using namespace lbk;

extern "C" size_t lbk_moe_route_ints(size_t n, size_t experts, size_t top) { return moe_route_ints(n, experts, top); }

extern "C" int lbk_moe_route(lbk_ctx *c, const float *z_dev, size_t z_pitch, size_t n, size_t experts, size_t top, int32_t *scratch_dev, const uint16_t *x_dev,
                             size_t x_pitch, uint16_t *sorted_dev, int32_t *ids_out_dev, float *weights_out_dev, int32_t *place_out_dev,
                             int32_t *offs_out_dev, void *stream) {
    if (!c) return fail(LBK_ERR_INVALID, "lbk_moe_route: context is null");
    if (n && (!z_dev || !scratch_dev || (sorted_dev && !x_dev))) return fail(LBK_ERR_INVALID, "lbk_moe_route: null buffer");
    if (sorted_dev && x_pitch % 64) return fail(LBK_ERR_SHAPE, "lbk_moe_route: rows of a multiple of 64 values");
    Ctx *ctx = reinterpret_cast<Ctx *>(c);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    LBK_CUDA(cudaSetDevice(ctx->device));
    MoeRoute r;
    moe_route_carve(r, scratch_dev, n, experts, top);
    LBK_CUDA(cudaMemsetAsync(r.counts, 0, kMaxExperts * 4, st));
    LBK_TRY(launch_moe_route(ctx, z_dev, static_cast<long>(z_pitch), n, experts, top, r, x_dev, static_cast<long>(x_pitch), sorted_dev, st));
    if (ids_out_dev) LBK_CUDA(cudaMemcpyAsync(ids_out_dev, r.ids, n * top * 4, cudaMemcpyDeviceToDevice, st));
    if (weights_out_dev) LBK_CUDA(cudaMemcpyAsync(weights_out_dev, r.weight, n * top * 4, cudaMemcpyDeviceToDevice, st));
    if (place_out_dev) LBK_CUDA(cudaMemcpyAsync(place_out_dev, r.place, n * top * 4, cudaMemcpyDeviceToDevice, st));
    if (offs_out_dev) LBK_CUDA(cudaMemcpyAsync(offs_out_dev, r.offs, (experts + 1) * 4, cudaMemcpyDeviceToDevice, st));
    return LBK_OK;
}

// Per-token absmax int8 activation quantiser, standalone form.
//
// Replaces quantize_acts / quantize_acts_into / quantize_row_scalar / quantize_row_avx2
// (crates/lb-ternary/src/quant.rs:37-193): one CTA per token row computes
// scale = 127/max(amax,1e-5), q = clamp(round_half_even(x*scale)), sum(q), and writes q
// zero padded to padded_cols(k). The decode GEMV has its own fused copy of this; this
// kernel feeds the prefill GEMM and the quantize_acts entry point.
#include "lbk_internal.cuh"
#include "lbk_ptx.cuh"

namespace lbk {

namespace {

__device__ __forceinline__ int quant_one(float v, float scale) {
    int r = __float2int_rn(__fmul_rn(v, scale));  // NaN -> 0 like `NaN as i8` (quant.rs:115-118)
    return max(-128, min(127, r));
}

// One CTA of T threads per row. ROW: float4 a thread holds between the maximum and the rounding (rows of up to 4 T ROW values,
// 16-byte aligned, are read once), 0: any row, read twice. A thread holds what the row needs and no more: with 8 for every row four
// CTAs fit an SM instead of eight. Bound: HBM. 2048 rows of 2560 / 4096 / 6912: 8.4 -> 6.2, 9.8 -> 7.9, 12.1 -> 11.3 us (4.2 to 6.2 TB/s); of 14336, read
// twice before, 35.1 -> 27.1 (5.4 TB/s). 512 threads for 6912 values took 13.7, 1024 18.3. It starts beside the end of the kernel in front (11 rows of 2560: 1.9 -> 1.6).
// amax_in: per-row max|x| supplied by the caller (tensor-parallel: the maximum over all ranks'
// column slices), or null to compute it here. amax_out: when non-null only the row maximum is
// written and nothing is quantised.
template <int T, int ROW>
__global__ void __launch_bounds__(T) quantize_kernel(const float *x, int k,
                                                            int kp, int8_t *__restrict__ q,
                                                            float *__restrict__ scale,
                                                            int32_t *__restrict__ sum,
                                                            const float *amax_in,
                                                            float *__restrict__ amax_out) {
    __shared__ float s_f[T / 32];
    __shared__ int s_i[T / 32];
    __shared__ float s_scale;
    // A kernel launched behind this one with programmatic stream serialisation (the prefill GEMM)
    // may start its prologue now; it waits for this grid's results with griddepcontrol.wait.
    ptx::pdl_trigger();
    ptx::pdl_wait();  // x may come from the kernel in front, and the rows of codes may still be read by it
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *xr = x + static_cast<size_t>(row) * k;
    int8_t *qr = q + static_cast<size_t>(row) * kp;
    const bool vec = (k & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;

    constexpr bool cached = ROW != 0;
    constexpr int kBatch = 4;  // 8: 2048 rows of 2561 8.1 -> 10.3 us
    float4 cache[cached ? ROW : 1];
    const int n4 = k >> 2;
    float am = 0.0f;  // fmaxf drops a NaN operand, as f32::max does (quant.rs:101-104)
    if constexpr (cached) {
        const float4 *x4 = reinterpret_cast<const float4 *>(xr);
#pragma unroll
        for (int j = 0; j < ROW; ++j) {
            const int i = tid + j * T;
            cache[j] = i < n4 ? __ldcg(x4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (amax_in == nullptr) {
#pragma unroll
            for (int j = 0; j < ROW; ++j)
                am = fmaxf(am, fmaxf(fmaxf(fabsf(cache[j].x), fabsf(cache[j].y)), fmaxf(fabsf(cache[j].z), fabsf(cache[j].w))));
        }
    }
    if (amax_in != nullptr) {
        am = __ldcg(amax_in + row);
    } else if (cached) {
        // done above
    } else if (vec) {
        const float4 *x4 = reinterpret_cast<const float4 *>(xr);
        for (int i0 = tid; i0 < n4; i0 += kBatch * T) {
            float4 v[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) v[j] = i0 + j * T < n4 ? x4[i0 + j * T] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < kBatch; ++j) am = fmaxf(am, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
        }
    } else {
        for (int i0 = tid; i0 < k; i0 += 2 * kBatch * T) {
            float v[2 * kBatch];
#pragma unroll
            for (int j = 0; j < 2 * kBatch; ++j) v[j] = i0 + j * T < k ? xr[i0 + j * T] : 0.0f;
#pragma unroll
            for (int j = 0; j < 2 * kBatch; ++j) am = fmaxf(am, fabsf(v[j]));
        }
    }
    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (lane == 0) s_f[warp] = am;
    __syncthreads();
    if (tid == 0) {
        float a = 0.0f;
        for (int w = 0; w < T / 32; ++w) a = fmaxf(a, s_f[w]);
        if (amax_out != nullptr) amax_out[row] = a;
        s_scale = __fdiv_rn(127.0f, fmaxf(a, 1e-5f));
    }
    __syncthreads();
    if (amax_out != nullptr) return;
    const float sc = s_scale;
    int acc = 0;
    if constexpr (cached) {
#pragma unroll
        for (int j = 0; j < ROW; ++j) {
            const int i = (tid + j * T) * 4;
            if (i < kp) {  // columns past k hold zeros, which quantise to zero
                const int q0 = quant_one(cache[j].x, sc), q1 = quant_one(cache[j].y, sc);
                const int q2 = quant_one(cache[j].z, sc), q3 = quant_one(cache[j].w, sc);
                acc += q0 + q1 + q2 + q3;
                *reinterpret_cast<uint32_t *>(qr + i) = (q0 & 255) | ((q1 & 255) << 8) | ((q2 & 255) << 16) |
                                                        (static_cast<uint32_t>(q3 & 255) << 24);
            }
        }
        for (int i = (tid + ROW * T) * 4; i < kp; i += T * 4) *reinterpret_cast<uint32_t *>(qr + i) = 0u;
    } else {
        // The second time a row comes from L1 or L2, by plain loads: what the kernel in front wrote is visible behind the wait. Both times a batch is asked for
        // together, which the compiler does not do around the stores. Past L1 and one load at a time 11 rows of 20000 / 2561 took 9.4 / 3.7 us, now
        // 4.5 / 2.3, 2048 rows of 20000 58.1, now 46.9.
        for (int i0 = tid * 4; i0 < kp; i0 += kBatch * T * 4) {
            float v[kBatch][4];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int i = i0 + j * T * 4;
                if (vec) {
                    const float4 f = i < k ? *reinterpret_cast<const float4 *>(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[j][0] = f.x; v[j][1] = f.y; v[j][2] = f.z; v[j][3] = f.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[j][e] = i + e < k ? xr[i + e] : 0.0f;
                }
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int i = i0 + j * T * 4;
                if (i >= kp) break;
                const int q0 = quant_one(v[j][0], sc), q1 = quant_one(v[j][1], sc), q2 = quant_one(v[j][2], sc), q3 = quant_one(v[j][3], sc);
                acc += q0 + q1 + q2 + q3;
                *reinterpret_cast<uint32_t *>(qr + i) = (q0 & 255) | ((q1 & 255) << 8) | ((q2 & 255) << 16) | (static_cast<uint32_t>(q3 & 255) << 24);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) s_i[warp] = acc;
    __syncthreads();
    if (tid == 0) {
        int s = 0;
        for (int w = 0; w < T / 32; ++w) s += s_i[w];
        scale[row] = sc;
        sum[row] = s;
    }
}

// y[t, r] = (float)dot[t, r] * (1 / (s_a[t] * s_w)): the epilogue of gemm.rs:141,158 as a kernel
// of its own, for dots that were summed across ranks first.
__global__ void __launch_bounds__(256) scale_epilogue_kernel(const int32_t *__restrict__ dots,
                                                            const float *__restrict__ ascale, float wscale,
                                                            int rows, size_t total, float *__restrict__ out) {
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const float inv = __fdiv_rn(1.0f, __fmul_rn(ascale[i / rows], wscale));
        out[i] = __fmul_rn(__int2float_rn(dots[i]), inv);
    }
}

// The same for up to LBK_MAX_GROUP matrices that share the token rows, in one launch (blockIdx.y is
// the matrix). `clean`: the sums live in the context's own accumulation buffer, which is kept zero
// between launches: every word is zeroed again once it has been read.
struct EpilogueGroup {
    int32_t *dots[LBK_MAX_GROUP];
    float *out[LBK_MAX_GROUP];
    float wscale[LBK_MAX_GROUP];
    int rows[LBK_MAX_GROUP];
    int clean[LBK_MAX_GROUP];
};
__global__ void __launch_bounds__(256) scale_epilogue_group_kernel(const EpilogueGroup g, const float *__restrict__ ascale, int m) {
    const int mat = blockIdx.y, rows = g.rows[mat];
    int32_t *dots = g.dots[mat];
    float *out = g.out[mat];
    if (!out) return;
    const float ws = g.wscale[mat];
    const size_t total = static_cast<size_t>(m) * rows;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const float inv = __fdiv_rn(1.0f, __fmul_rn(ascale[i / rows], ws));
        out[i] = __fmul_rn(__int2float_rn(dots[i]), inv);
        if (g.clean[mat]) dots[i] = 0;
    }
}

}  // namespace

int launch_scale_epilogue_group(Ctx *ctx, int n, int32_t *const *dots, float *const *outs, const float *wscale, const int *rows, const bool *clean,
                                const float *ascale, size_t m, cudaStream_t stream) {
    EpilogueGroup g{};
    size_t most = 0;
    for (int i = 0; i < n; ++i) {
        g.dots[i] = dots[i];
        g.out[i] = outs[i];
        g.wscale[i] = wscale[i];
        g.rows[i] = rows[i];
        g.clean[i] = clean[i] ? 1 : 0;
        if (outs[i] && m * static_cast<size_t>(rows[i]) > most) most = m * static_cast<size_t>(rows[i]);
    }
    if (most == 0) return LBK_OK;
    size_t blocks = (most + 255) / 256;
    if (blocks > static_cast<size_t>(ctx->sm_count) * 8) blocks = static_cast<size_t>(ctx->sm_count) * 8;
    scale_epilogue_group_kernel<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(n)), 256, 0, stream>>>(g, ascale, static_cast<int>(m));
    LBK_CUDA(cudaGetLastError());
    ctx->launches++;
    return LBK_OK;
}

int launch_scale_epilogue(Ctx *ctx, const int32_t *dots, const float *ascale, float wscale, size_t m, size_t rows,
                          float *out, cudaStream_t stream) {
    const size_t total = m * rows;
    if (total == 0) return LBK_OK;
    size_t blocks = (total + 255) / 256;
    if (blocks > static_cast<size_t>(ctx->sm_count) * 8) blocks = static_cast<size_t>(ctx->sm_count) * 8;
    scale_epilogue_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(dots, ascale, wscale, static_cast<int>(rows), total, out);
    LBK_CUDA(cudaGetLastError());
    ctx->launches++;
    return LBK_OK;
}

int launch_quantize_ex(Ctx *ctx, const float *x, size_t m, size_t k, int8_t *q, float *scale, int32_t *sum,
                       const float *amax_in, float *amax_out, cudaStream_t stream) {
    if (m == 0) return LBK_OK;
    const size_t kp = lbk_padded_cols(k), n4 = k / 4;
    const bool vec = k % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    void (*kernel)(const float *, int, int, int8_t *, float *, int32_t *, const float *, float *) = quantize_kernel<256, 0>;
    unsigned threads = 256;
    if (vec && n4 <= 3 * 256) kernel = quantize_kernel<256, 3>;
    else if (vec && n4 <= 4 * 256) kernel = quantize_kernel<256, 4>;
    else if (vec && n4 <= 7 * 256) kernel = quantize_kernel<256, 7>;
    // 2048 rows of 8192 / 8640 / 12288 by 512 threads, half of what they hold empty, 17.6 / 18.6 / 25.2 us, by 256 11.2 / 12.7 / 20.9; one or two rows an SM in
    // front of a GEMM are done sooner by 512 (128 rows of 8192 -> 8192 14.5 us with the GEMM, by 256 15.0)
    else if (vec && n4 <= 8 * 256 && m > 2 * static_cast<size_t>(ctx->sm_count)) kernel = quantize_kernel<256, 8>;
    else if (vec && n4 <= 12 * 256 && m > 2 * static_cast<size_t>(ctx->sm_count)) kernel = quantize_kernel<256, 12>;
    else if (vec && n4 <= 8 * 512) kernel = quantize_kernel<512, 8>, threads = 512;
    // Rows read twice that together do not fit in L2 with eight CTAs an SM (135 MB of 28672 values) come in fours: shared memory that nobody uses.
    const size_t smem = k > 21000 && m > 4 * static_cast<size_t>(ctx->sm_count) ? 47 * 1024 : 0;
    LBK_CUDA(launch_chained(kernel, dim3(static_cast<unsigned>(m)), dim3(threads), smem, stream, x, static_cast<int>(k), static_cast<int>(kp), q, scale, sum, amax_in, amax_out));
    LBK_CUDA(cudaGetLastError());
    ctx->launches++;
    return LBK_OK;
}

int launch_quantize(Ctx *ctx, const float *x, size_t m, size_t k, int8_t *q, float *scale,
                    int32_t *sum, cudaStream_t stream) {
    return launch_quantize_ex(ctx, x, m, k, q, scale, sum, nullptr, nullptr, stream);
}

}  // namespace lbk

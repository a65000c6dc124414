// Q8_0 activation quantizer kernels, alone and fused behind RMSNorm / SiLU*mul.
#include "act.cuh"
#include "ops.h"

namespace cera {

namespace {

// One warp per (column, block).  strided != 0: x is [k x n] with row stride n.
__global__ void quantize_kernel(const float *__restrict__ x, size_t k, size_t n, int strided, float *scales,
                                int8_t *quants, int16_t *sums) {
    pdl_trigger();
    pdl_wait();
    const size_t nb = k / 32;
    const size_t wid = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= nb * n) return;
    const size_t j = wid / nb, b = wid % nb;
    const size_t e = b * 32 + lane;
    const float v = strided ? x[e * n + j] : x[j * k + e];
    float scale;
    int hs;
    const int q = quantize_lane(v, scale, hs);
    quants[j * k + e] = (int8_t)q;
    if (lane == 0) scales[j * nb + b] = scale;
    if (sums && (lane & 15) == 0) sums[j * (k / 16) + b * 2 + (lane >> 4)] = (int16_t)hs;
}

// The same for contiguous columns, a thread per four consecutive elements: one 128-bit load and eight lanes a block, where a warp per
// block had one 4-byte load in flight per thread.  n_vec = k / 4 * n, a multiple of 8.
// The product behind it may be launched once the work is done: placed while these blocks still fill the SMs, the clusters of a small batch share SMs that they
// would have to themselves (4096 x 4096 Q4_K, 12 columns: 25.6 us, 17.4 so; 4096 x 14336 Q6_K, 40 columns: 120 and 103).
__global__ void __launch_bounds__(256) quantize_quad_kernel(const float *__restrict__ x, size_t n_vec, float *scales, int8_t *quants, int16_t *sums) {
    pdl_wait();
    const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = v < n_vec;  // a block's eight lanes are all in or all out
    const float4 x4 = in ? reinterpret_cast<const float4 *>(x)[v] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float e[4] = {x4.x, x4.y, x4.z, x4.w};
    const QuantQuad o = quantize_quad(e);
    if (in) {
        reinterpret_cast<uint32_t *>(quants)[v] = o.quants;
        if ((threadIdx.x & 7) == 0) scales[v >> 3] = o.scale;
        if (sums && (threadIdx.x & 3) == 0) sums[v >> 2] = (int16_t)o.half_sum;
    }
    pdl_trigger();
}

// RMSNorm of one column per CTA (cera/src/backend/cpu.rs:2479-2496: f64 sum of
// squares, inv = (float)(1/sqrt(mean+eps)), x*inv*w left to right), then
// optionally the Q8_0 quantizer on the normed values.  Latency-bound and on the critical path of
// every projection: 32 warps, every thread's x and w values fetched once with all loads issued
// before the reduction, and at most four 32-element blocks quantized per warp one after another
// (up to 4096 elements; longer columns loop).
constexpr int RN_WARPS = 32, RN_THREADS = RN_WARPS * 32, RN_CH = 4;

__global__ void __launch_bounds__(RN_THREADS) rmsnorm_kernel(const float *__restrict__ x, const float *__restrict__ weight,
                                                              size_t n_elem, double inv_n, float eps, float *out_f32,
                                                              float *scales, int8_t *quants, int16_t *sums, const TpHook tp) {
    __shared__ double red[RN_WARPS];
    __shared__ float inv_s;
    pdl_trigger();
    const size_t col = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nblk = (uint32_t)((n_elem + 31) >> 5);
    const bool single = nblk <= RN_WARPS * RN_CH;  // up to 4096 elements stay in registers
    // lane `lane` of warp `warp` owns element `lane` of 32-blocks warp, warp+32, ...
    float wv[RN_CH], xv[RN_CH];
    if (single) {
#pragma unroll
        for (int j = 0; j < RN_CH; ++j) {
            const size_t i = (size_t)(warp + RN_WARPS * j) * 32 + lane;
            wv[j] = i < n_elem ? weight[i] : 0.0f;  // weights do not depend on the previous kernel
        }
    }
    pdl_wait();
    tp_arrive_wait(tp.ctx, tp.wait_slot);
    const float *xc = x + col * n_elem;
    double ss = 0.0;
    for (uint32_t c0 = 0; c0 < nblk; c0 += RN_WARPS * RN_CH) {
#pragma unroll
        for (int j = 0; j < RN_CH; ++j) {
            const size_t i = (size_t)(c0 + warp + RN_WARPS * j) * 32 + lane;
            xv[j] = i < n_elem ? xc[i] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < RN_CH; ++j) ss += (double)xv[j] * (double)xv[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    if (warp == 0) {
        double t = red[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) inv_s = (float)(1.0 / sqrt(t / (double)n_elem + (double)eps));  // the reference's f64 expression, IEEE division and square root
    }
    __syncthreads();
    const float inv = inv_s;
    for (uint32_t c0 = 0; c0 < nblk; c0 += RN_WARPS * RN_CH) {
#pragma unroll
        for (int j = 0; j < RN_CH; ++j) {
            const uint32_t b = c0 + warp + RN_WARPS * j;
            if (b >= nblk) continue;  // warp-uniform
            const size_t i = (size_t)b * 32 + lane;
            const bool in = i < n_elem;  // only the f32-only path may see a ragged last block
            const float xi = single ? xv[j] : (in ? xc[i] : 0.0f);
            const float wi = single ? wv[j] : (in ? weight[i] : 0.0f);
            const float v = __fmul_rn(__fmul_rn(xi, inv), wi);
            if (out_f32 && in) out_f32[col * n_elem + i] = v;
            if (quants) {
                float scale;
                int hs;
                const int q = quantize_lane(v, scale, hs);
                quants[col * n_elem + i] = (int8_t)q;
                if (lane == 0) scales[col * (n_elem / 32) + b] = scale;
                if ((lane & 15) == 0) sums[col * (n_elem / 16) + 2 * b + (lane >> 4)] = (int16_t)hs;
            }
        }
    }
}

// The same operation for columns whose length is a multiple of 32.  1024 virtual threads own FOUR consecutive elements each (one 128-bit
// load of x and of the weights), so a 32-element Q8_0 block is eight neighbouring lanes and all blocks of the column are quantized at the same
// time.  Up to 4096 elements stay in registers between the sum of squares and the scaling; longer columns re-read x.
// The CTA's warps share the 32 virtual ones; sums are added in the same order whatever their number.  One column is latency: 32 warps (eight:
// 0.6 us more in a decode step).  Many columns are throughput, and a CTA of 32 warps holds two of an SM's columns at a time while most of its warps
// wait for the scale: eight warps, five columns.  2047 x 4096: 64 -> 21 us, 600 x 4096 17.4 -> 8.6, 149 x 4096 7.1 both, 149 x 1024 7.0 -> 5.1.
template <int RQ_WARPS>
__global__ void __launch_bounds__(RQ_WARPS * 32, RQ_WARPS == RN_WARPS ? 1 : 5) rmsnorm_q8_kernel(const float *__restrict__ x, const float *__restrict__ weight, size_t n_elem, float eps,
                                                                float *out_f32, float *scales, int8_t *quants, int16_t *sums, const TpHook tp) {
    constexpr int VT = RN_THREADS, PER = RN_WARPS / RQ_WARPS;  // virtual threads; of a thread
    __shared__ double red[RN_WARPS];
    __shared__ float inv_s;
    pdl_trigger();
    const size_t col = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nvec = (uint32_t)(n_elem >> 2);
    const bool single = nvec <= VT;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 wv[PER], xv[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t v = threadIdx.x + j * RQ_WARPS * 32;
        wv[j] = single && v < nvec ? reinterpret_cast<const float4 *>(weight)[v] : zero;  // independent of the previous kernel
    }
    pdl_wait();
    tp_arrive_wait(tp.ctx, tp.wait_slot);
    const float4 *xc = reinterpret_cast<const float4 *>(x + col * n_elem);
    double ss[PER] = {};
    for (uint32_t v0 = 0; v0 < nvec; v0 += VT) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t v = v0 + threadIdx.x + j * RQ_WARPS * 32;
            xv[j] = v < nvec ? xc[v] : zero;
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (v0 + threadIdx.x + j * RQ_WARPS * 32 >= nvec) continue;
            ss[j] += (double)xv[j].x * (double)xv[j].x;
            ss[j] += (double)xv[j].y * (double)xv[j].y;
            ss[j] += (double)xv[j].z * (double)xv[j].z;
            ss[j] += (double)xv[j].w * (double)xv[j].w;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < PER; ++j) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], o);
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < PER; ++j) red[warp + j * RQ_WARPS] = ss[j];
    __syncthreads();
    if (warp == 0) {
        double t = red[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) inv_s = (float)(1.0 / sqrt(t / (double)n_elem + (double)eps));  // the reference's f64 expression, IEEE division and square root
    }
    __syncthreads();
    const float inv = inv_s;
    // whole warps iterate together: nvec is a multiple of 8, so a block's eight lanes are all in or all out
    for (uint32_t v0 = 0; v0 < nvec; v0 += VT)
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const uint32_t v = v0 + threadIdx.x + j * RQ_WARPS * 32;
            const bool in = v < nvec;
            const float4 xi = single ? xv[j] : in ? xc[v] : zero, wi = single ? wv[j] : in ? reinterpret_cast<const float4 *>(weight)[v] : zero;
            const float e[4] = {__fmul_rn(__fmul_rn(xi.x, inv), wi.x), __fmul_rn(__fmul_rn(xi.y, inv), wi.y), __fmul_rn(__fmul_rn(xi.z, inv), wi.z),
                                __fmul_rn(__fmul_rn(xi.w, inv), wi.w)};
            if (out_f32 && in) reinterpret_cast<float4 *>(out_f32 + col * n_elem)[v] = make_float4(e[0], e[1], e[2], e[3]);
            const QuantQuad o = quantize_quad(e);
            if (in) {
                reinterpret_cast<uint32_t *>(quants + col * n_elem)[v] = o.quants;
                if ((lane & 7) == 0) scales[col * (n_elem / 32) + (v >> 3)] = o.scale;
                if ((lane & 3) == 0) sums[col * (n_elem / 16) + (v >> 2)] = (int16_t)o.half_sum;
            }
        }
}

__global__ void silu_mul_kernel(float *gate, const float *__restrict__ up, size_t n_elem, size_t n_cols,
                                float *scales, int8_t *quants, int16_t *sums, const TpHook tp) {
    pdl_trigger();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_elem * n_cols) return;
    const float v = silu_mul(gate[i], up[i]);
    gate[i] = v;
    if (quants) {
        float scale;
        int hs;
        const int q = quantize_lane(v, scale, hs);
        const int lane = threadIdx.x & 31;
        quants[i] = (int8_t)q;
        if (lane == 0) scales[i / 32] = scale;
        if ((lane & 15) == 0) sums[i / 16] = (int16_t)hs;
        if (tp.push) {
            tp_push(tp.ctx, quants + i, (int8_t)q);
            if (lane == 0) tp_push(tp.ctx, scales + i / 32, scale);
            if ((lane & 15) == 0) tp_push(tp.ctx, sums + i / 16, (int16_t)hs);
        }
    }
}

// SiLU*mul with the Q8_0 quantizer, four consecutive elements per thread (one 128-bit load of gate and of up): a
// 32-element block is eight neighbouring lanes, so its amax takes three shuffle steps and its 16-element sums two.  keep: the
// product replaces gate (a third of the traffic, which a prompt's product on the quants alone does without).
__global__ void __launch_bounds__(256) silu_mul_q8_kernel(float *gate, const float *__restrict__ up, size_t n_vec, int keep, float *scales,
                                                          int8_t *quants, int16_t *sums, const TpHook tp) {
    pdl_trigger();
    pdl_wait();
    const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = v < n_vec;  // n_vec is a multiple of 8: a block's eight lanes are all in or all out
    const int lane = threadIdx.x & 31;
    float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f), u4 = g4;
    if (in) {
        g4 = reinterpret_cast<const float4 *>(gate)[v];
        u4 = reinterpret_cast<const float4 *>(up)[v];
    }
    const float e[4] = {silu_mul(g4.x, u4.x), silu_mul(g4.y, u4.y), silu_mul(g4.z, u4.z), silu_mul(g4.w, u4.w)};
    if (in && keep) reinterpret_cast<float4 *>(gate)[v] = make_float4(e[0], e[1], e[2], e[3]);
    const QuantQuad o = quantize_quad(e);
    if (!in) return;
    reinterpret_cast<uint32_t *>(quants)[v] = o.quants;
    if ((lane & 7) == 0) scales[v >> 3] = o.scale;
    if ((lane & 3) == 0) sums[v >> 2] = (int16_t)o.half_sum;
    if (tp.push) {
        tp_push(tp.ctx, reinterpret_cast<uint32_t *>(quants) + v, o.quants);
        if ((lane & 7) == 0) tp_push(tp.ctx, scales + (v >> 3), o.scale);
        if ((lane & 3) == 0) tp_push(tp.ctx, sums + (v >> 2), (int16_t)o.half_sum);
    }
}

// The same, eight elements per thread, for a prompt's columns.  What bounds it: instructions and the pipe that shuffles and reciprocals share (four
// elements: 300 a thread, a third of the stalls there).  512 x 14336: 29 us with four elements, 13.6 now; 2047: 114 and 53.
__global__ void __launch_bounds__(256) silu_mul_q8_wide_kernel(float4 *gate, const float4 *__restrict__ up, size_t n_oct, int keep, float *scales, uint2 *quants, int16_t *sums) {
    pdl_trigger();
    pdl_wait();
    const size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = v < n_oct;  // n_oct is a multiple of 4: a block's four lanes are all in or all out
    float4 g[2] = {}, u[2] = {};
    if (in) {
#pragma unroll
        for (int i = 0; i < 2; ++i) g[i] = gate[2 * v + i], u[i] = up[2 * v + i];
    }
    float e[8];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float2 a = silu_mul2(make_float2(g[i].x, g[i].y), make_float2(u[i].x, u[i].y)), b = silu_mul2(make_float2(g[i].z, g[i].w), make_float2(u[i].z, u[i].w));
        e[4 * i] = a.x, e[4 * i + 1] = a.y, e[4 * i + 2] = b.x, e[4 * i + 3] = b.y;
        if (in && keep) gate[2 * v + i] = make_float4(a.x, a.y, b.x, b.y);
    }
    const QuantOct o = quantize_oct(e);
    if (!in) return;
    quants[v] = o.quants;
    if ((threadIdx.x & 3) == 0) scales[v >> 2] = o.scale;
    if ((threadIdx.x & 1) == 0) sums[v >> 1] = (int16_t)o.half_sum;
}

}  // namespace

int32_t launch_quantize(const float *x, size_t k, size_t n, bool strided, float *scales, int8_t *quants,
                        int16_t *sums, cudaStream_t st) {
    if (!x || !scales || !quants) return fail(CERA_CUDA_ERR_BAD_ARG, "quantize_q8_0: null argument");
    if (k == 0 || k % 32) return fail(CERA_CUDA_ERR_BAD_ARG, "quantize_q8_0: k=%zu must be a positive multiple of 32", k);
    if (n == 0) return CERA_CUDA_OK;
    const int threads = 256;
    if (!strided && (uintptr_t)x % 16 == 0 && (uintptr_t)quants % 4 == 0) {
        const size_t n_vec = k / 4 * n;
        CERA_CUDA_TRY(launch_k(quantize_quad_kernel, dim3((unsigned)((n_vec + threads - 1) / threads)), dim3(threads), 0, st, x, n_vec, scales, quants, sums));
        count_launch();
        return check_cuda(cudaGetLastError(), "quantize launch");
    }
    const size_t warps = (k / 32) * n;
    const size_t grid = (warps * 32 + threads - 1) / threads;
    CERA_CUDA_TRY(launch_k(quantize_kernel, dim3((unsigned)grid), dim3(threads), 0, st, x, k, n, strided ? 1 : 0, scales, quants, sums));
    count_launch();
    return check_cuda(cudaGetLastError(), "quantize launch");
}

int32_t launch_rmsnorm(const float *x, const float *weight, size_t n_elem, size_t n_cols, float eps, float *out_f32,
                       float *scales, int8_t *quants, int16_t *sums, cudaStream_t st, const TpHook *tp) {
    if (!x || !weight) return fail(CERA_CUDA_ERR_BAD_ARG, "rmsnorm: null argument");
    if (quants && (n_elem % 32 || !scales || !sums))
        return fail(CERA_CUDA_ERR_BAD_ARG, "rmsnorm+quantize: n=%zu must be a multiple of 32", n_elem);
    if (n_elem == 0 || n_cols == 0) return CERA_CUDA_OK;
    const int threads = RN_THREADS;
    if (quants && ((uintptr_t)x % 16 == 0) && ((uintptr_t)weight % 16 == 0) && (!out_f32 || (uintptr_t)out_f32 % 16 == 0) &&
        (uintptr_t)quants % 4 == 0) {
        const TpHook hook = tp ? *tp : TpHook{};
        if (n_cols > (size_t)sm_count())
            CERA_CUDA_TRY(launch_k(rmsnorm_q8_kernel<8>, dim3((unsigned)n_cols), dim3(256), 0, st, x, weight, n_elem, eps, out_f32, scales, quants, sums, hook));
        else
            CERA_CUDA_TRY(launch_k(rmsnorm_q8_kernel<RN_WARPS>, dim3((unsigned)n_cols), dim3(threads), 0, st, x, weight, n_elem, eps, out_f32, scales, quants,
                                   sums, hook));
        count_launch();
        return check_cuda(cudaGetLastError(), "rmsnorm launch");
    }
    CERA_CUDA_TRY(launch_k(rmsnorm_kernel, dim3((unsigned)n_cols), dim3(threads), 0, st, x, weight, n_elem, 1.0 / (double)n_elem, eps, out_f32, scales,
                           quants, sums, tp ? *tp : TpHook{}));
    count_launch();
    return check_cuda(cudaGetLastError(), "rmsnorm launch");
}

int32_t launch_silu_mul(float *gate, const float *up, size_t n_elem, size_t n_cols, float *scales, int8_t *quants,
                        int16_t *sums, cudaStream_t st, const TpHook *tp, bool keep) {
    if (!gate || !up) return fail(CERA_CUDA_ERR_BAD_ARG, "silu_mul: null argument");
    if (quants && n_elem % 32) return fail(CERA_CUDA_ERR_BAD_ARG, "silu_mul+quantize: n=%zu must be a multiple of 32", n_elem);
    const size_t total = n_elem * n_cols;
    if (total == 0) return CERA_CUDA_OK;
    const int threads = 256;
    if (quants && (uintptr_t)gate % 16 == 0 && (uintptr_t)up % 16 == 0 && (uintptr_t)quants % 4 == 0) {
        const size_t n_vec = total / 4;
        // the wide one once its threads fill the device (fewer columns leave a thread's chain of work as the time)
        if (total / 8 >= (size_t)sm_count() * 2048 && !(tp && tp->push) && (uintptr_t)quants % 8 == 0) {
            count_launch();
            return check_cuda(launch_k(silu_mul_q8_wide_kernel, dim3((unsigned)((total / 8 + threads - 1) / threads)), dim3(threads), 0, st, (float4 *)gate,
                                       (const float4 *)up, total / 8, keep ? 1 : 0, scales, (uint2 *)quants, sums),
                              "silu_mul launch");
        }
        CERA_CUDA_TRY(launch_k(silu_mul_q8_kernel, dim3((unsigned)((n_vec + threads - 1) / threads)), dim3(threads), 0, st, gate, up, n_vec,
                               keep ? 1 : 0, scales, quants, sums, tp ? *tp : TpHook{}));
        count_launch();
        return check_cuda(cudaGetLastError(), "silu_mul launch");
    }
    CERA_CUDA_TRY(launch_k(silu_mul_kernel, dim3((unsigned)((total + threads - 1) / threads)), dim3(threads), 0, st, gate, up,
                           n_elem, n_cols, scales, quants, sums, tp ? *tp : TpHook{}));
    count_launch();
    return check_cuda(cudaGetLastError(), "silu_mul launch");
}

}  // namespace cera

using namespace cera;

extern "C" {

int32_t cera_cuda_quantize_q8_0(const float *x_dev, size_t k, size_t n, float *scales_dev, int8_t *quants_dev,
                                int16_t *sums_dev, void *stream) {
    return launch_quantize(x_dev, k, n, false, scales_dev, quants_dev, sums_dev, (cudaStream_t)stream);
}

int32_t cera_cuda_quantize_columns(const float *mat_dev, size_t dim, size_t n, float *scales_dev, int8_t *quants_dev,
                                   int16_t *sums_dev, void *stream) {
    return launch_quantize(mat_dev, dim, n, true, scales_dev, quants_dev, sums_dev, (cudaStream_t)stream);
}

int32_t cera_cuda_rmsnorm(const float *x_dev, const float *weight_dev, size_t n, float eps, float *out_dev,
                          void *stream) {
    if (!out_dev) return fail(CERA_CUDA_ERR_BAD_ARG, "rmsnorm: null output");
    return launch_rmsnorm(x_dev, weight_dev, n, 1, eps, out_dev, nullptr, nullptr, nullptr, (cudaStream_t)stream);
}

int32_t cera_cuda_rmsnorm_q8_0(const float *x_dev, const float *weight_dev, size_t n, float eps, float *out_dev,
                               float *scales_dev, int8_t *quants_dev, int16_t *sums_dev, void *stream) {
    if (!scales_dev || !quants_dev || !sums_dev) return fail(CERA_CUDA_ERR_BAD_ARG, "rmsnorm_q8_0: null output");
    return launch_rmsnorm(x_dev, weight_dev, n, 1, eps, out_dev, scales_dev, quants_dev, sums_dev, (cudaStream_t)stream);
}

int32_t cera_cuda_silu_mul(float *gate_dev, const float *up_dev, size_t n, void *stream) {
    return launch_silu_mul(gate_dev, up_dev, n, 1, nullptr, nullptr, nullptr, (cudaStream_t)stream);
}

}  // extern "C"

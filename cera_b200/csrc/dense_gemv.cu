// One-column products with dense weights: the decode step's projections, with the work that follows them fused where
// one warp holds all a result needs (the minGRU update, the gated units, the sum over picks).
#include "dense_gemv.cuh"
#include "moe_route.cuh"

namespace cera {

namespace {

using namespace gv;

// Rows of this CTA's two units: gate, gate, up, up (an odd count's last pair repeats its unit).
template <class T>
__device__ __forceinline__ void unit_rows(const T *(&rows)[4], const T *w, uint32_t ff_p, uint32_t ld) {
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) rows[r] = w + (size_t)(min(blockIdx.x * 2 + (r & 1), ff_p - 1) + (r >> 1) * ff_p) * ld;
}

// A CTA per R rows, each shared by all its warps, two vectors of a row in flight per lane.  What bounds it: HBM.  Many warps that load
// little each keep it busier than few with long batches, whose later batches wait for the earlier ones' sums: 4096 x 8192 bf16
// 13.3 us (5.0 TB/s), 4096 x 4096 8.0, 18560 x 4096 24.1 (6.3 TB/s), 2048 x 2048 3.4; one row per two warps and eight vectors per
// lane: 18.1, 10.2, 25.8, 4.1.  R = 4 where that leaves every SM a CTA, R = 1 for fewer rows (a router's).
template <class T, int R>
__global__ void __launch_bounds__(GV_WARPS * 32) gemv_kernel(const T *__restrict__ w, uint32_t rows, uint32_t ld, const T *x, float *y) {
    __shared__ float red[GV_WARPS][R];
    pdl_trigger();
    const int warp = threadIdx.x >> 5;
    const uint32_t g = blockIdx.x;
    RowDot<T, R, R == 1 ? 8 : 2> d;
#pragma unroll
    for (int r = 0; r < R; ++r) d.w[r] = w + (size_t)min(g * R + r, rows - 1) * ld;
    d.start(ld, warp, GV_WARPS);
    d.fetch();
    pdl_wait();
    float acc[R] = {};
    d.run(x, acc);
    group_sum<R, GV_WARPS>(acc, red);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (g * R + r < rows) y[g * R + r] = acc[r];
    }
}

template <class T, int WPR>
__global__ void __launch_bounds__(GV_WARPS * 32) mingru_step_kernel(const T *__restrict__ w, uint32_t wp, uint32_t ld, const T *x,
                                                                    const float *__restrict__ zb, const float *__restrict__ xb, float *state, T *out) {
    __shared__ float red[GV_WARPS][3];
    pdl_trigger();
    const int warp = threadIdx.x >> 5;
    const uint32_t g = blockIdx.x * (GV_WARPS / WPR) + warp / WPR, gi = min(g, wp - 1);
    RowDot<T, 3, 4> d;
#pragma unroll
    for (int r = 0; r < 3; ++r) d.w[r] = w + (size_t)(gi + r * wp) * ld;
    d.start(ld, warp % WPR, WPR);
    d.fetch();
    pdl_wait();
    float acc[3] = {};
    d.run(x, acc);
    group_sum<3, WPR>(acc, red);
    if (warp % WPR == 0 && (threadIdx.x & 31) == 0 && g < wp) {
        float z, cand;
        mingru_gates(acc[0], acc[1], zb[g], xb[g], z, cand);
        const float s = (1.0f - z) * state[g] + z * cand;
        state[g] = s;
        out[g] = Elem<T>::from(s * silu_f32(acc[2]));
    }
}

// Rows [0, ff_p) gate, [ff_p, 2 ff_p) up of w; out = unit(gate, up).  A CTA per two units.
template <class T>
__global__ void __launch_bounds__(GV_WARPS * 32) gated_unit_step_kernel(const T *__restrict__ w, uint32_t ff_p, uint32_t ld, const T *x, ExpertAct a, T *out) {
    __shared__ float red[GV_WARPS][4];
    pdl_trigger();
    const int warp = threadIdx.x >> 5;
    RowDot<T, 4, 2> d;
    unit_rows(d.w, w, ff_p, ld);
    d.start(ld, warp, GV_WARPS);
    d.fetch();
    pdl_wait();
    float acc[4] = {};
    d.run(x, acc);
    group_sum<4, GV_WARPS>(acc, red);
    const uint32_t g = blockIdx.x * 2 + threadIdx.x;
    if (threadIdx.x < 2 && g < ff_p) out[g] = Elem<T>::from(gated_unit(threadIdx.x ? acc[1] : acc[0], threadIdx.x ? acc[3] : acc[2], a));
}

// grid (row groups, picks).  Every CTA repeats the pick from the router logits - few CTAs with long rows therefore (a CTA per two
// units: 17.7 us instead of 12.9, width 2048); CTA 0 of a pick leaves it for the down step.
template <class T, int WPR>
__global__ void __launch_bounds__(GV_WARPS * 32) expert_gate_up_kernel(const T *__restrict__ w, uint32_t ff_p, uint32_t ld, const T *x,
                                                                       const float *logits, RouterRule rule, ExpertAct a, uint32_t *ids,
                                                                       float *weights, T *act) {
    __shared__ float red[GV_WARPS][2];
    __shared__ float probs[MOE_MAX_EXPERTS];
    __shared__ uint32_t picked[MOE_MAX_USED];
    __shared__ float wt[MOE_MAX_USED];
    pdl_trigger();
    pdl_wait();
    for (uint32_t e = threadIdx.x; e < rule.n_expert; e += blockDim.x) probs[e] = logits[e];
    __syncthreads();
    moe_scores(probs, rule.n_expert, rule.softmax);
    const int warp = threadIdx.x >> 5;
    if (warp == 0) moe_pick(probs, nullptr, rule.n_expert, rule.n_used, rule.renorm, picked, wt);
    __syncthreads();
    const uint32_t s = blockIdx.y, e = picked[s];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ids[s] = e;
        weights[s] = wt[s];
    }
    const uint32_t g = blockIdx.x * (GV_WARPS / WPR) + warp / WPR, gi = min(g, ff_p - 1);
    RowDot<T, 2, 4> d;
    d.w[0] = w + ((size_t)e * 2 * ff_p + gi) * ld;
    d.w[1] = d.w[0] + (size_t)ff_p * ld;
    d.start(ld, warp % WPR, WPR);
    d.fetch();
    float acc[2] = {};
    d.run(x, acc);
    group_sum<2, WPR>(acc, red);
    if (warp % WPR == 0 && (threadIdx.x & 31) == 0 && g < ff_p) {
        const float sc = rule.weight_input ? wt[s] : 1.0f;
        act[(size_t)s * ff_p + g] = Elem<T>::from(gated_unit(sc * acc[0], sc * acc[1], a));
    }
}

// A CTA per R rows.  The picks' rows are walked as one row of n_used * ld elements, U vectors of it in flight per lane and row.
template <class T>
__global__ void __launch_bounds__(GV_WARPS * 32) expert_down_kernel(const T *__restrict__ w, uint32_t rows, uint32_t ld, const T *act, uint32_t n_used,
                                                                    int weight_input, const uint32_t *ids, const float *weights, float *y) {
    constexpr int R = 2, U = 4;
    __shared__ float red[GV_WARPS][R];
    pdl_trigger();
    pdl_wait();
    const uint32_t g = blockIdx.x * R, g1 = min(g + 1, rows - 1), nv = ld / Elem<T>::N, all = n_used * nv, step = 32u * GV_WARPS;
    float total[R] = {};
    for (uint32_t c = threadIdx.x; c < all; c += U * step) {
        uint4 wb[R][U], xb[U];
        float sc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t v = c + u * step, s = v / nv;
            if (v < all) {
                const T *expert = w + (size_t)ids[s] * rows * ld;
                wb[0][u] = ld_stream(reinterpret_cast<const uint4 *>(expert + (size_t)g * ld) + (v - s * nv));
                wb[1][u] = ld_stream(reinterpret_cast<const uint4 *>(expert + (size_t)g1 * ld) + (v - s * nv));
                xb[u] = *(reinterpret_cast<const uint4 *>(act) + v);
                sc[u] = weight_input ? 1.0f : weights[s];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c + u * step < all) {
                float xf[Elem<T>::N];
                Elem<T>::unpack(xb[u], xf);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float wf[Elem<T>::N], a = 0.0f;
                    Elem<T>::unpack(wb[r][u], wf);
#pragma unroll
                    for (int i = 0; i < Elem<T>::N; ++i) a = fmaf(wf[i], xf[i], a);
                    total[r] = fmaf(sc[u], a, total[r]);
                }
            }
    }
    group_sum<R, GV_WARPS>(total, red);
    if (threadIdx.x == 0) {
        y[g] = total[0];
        if (g + 1 < rows) y[g + 1] = total[1];
    }
}

}  // namespace

int32_t launch_dense_gemv(const DenseView &w, const void *x, float *y, cudaStream_t st) {
    const bool four = w.rows >= (uint32_t)sm_count() * 4;
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return check_cuda(four ? launch_k(gemv_kernel<T, 4>, dim3((w.rows + 3) / 4), dim3(GV_WARPS * 32), 0, st, (const T *)w.w, w.rows, w.ld, (const T *)x, y)
                               : launch_k(gemv_kernel<T, 1>, dim3(w.rows), dim3(GV_WARPS * 32), 0, st, (const T *)w.w, w.rows, w.ld, (const T *)x, y),
                          "dense gemv launch");
    });
}

int32_t launch_mingru_step(const DenseView &w, const void *x, const float *z_bias, const float *x_bias, float *state, void *out, cudaStream_t st) {
    const uint32_t wp = w.rows / 3;
    const int wpr = pick_wpr(wp, (size_t)w.ld * (w.f32 ? 4 : 2), 4);
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return with_wpr(wpr, [&](auto n) {
            return check_cuda(launch_k(mingru_step_kernel<T, decltype(n)::value>, gv_grid(wp, wpr), dim3(GV_WARPS * 32), 0, st, (const T *)w.w, wp, w.ld,
                                       (const T *)x, z_bias, x_bias, state, (T *)out),
                              "mingru step launch");
        });
    });
}

int32_t launch_gated_unit_step(const DenseView &w, const void *x, const ExpertAct &a, void *out, cudaStream_t st) {
    const uint32_t ff_p = w.rows / 2;
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return check_cuda(launch_k(gated_unit_step_kernel<T>, dim3((ff_p + 1) / 2), dim3(GV_WARPS * 32), 0, st, (const T *)w.w, ff_p, w.ld, (const T *)x, a, (T *)out),
                          "gated unit launch");
    });
}

int32_t launch_expert_gate_up_step(const DenseView &w, const void *x, const float *router_logits, const RouterRule &r, uint32_t ff_p, const ExpertAct &a,
                                   uint32_t *ids, float *weights, void *act, cudaStream_t st) {
    const int wpr = pick_wpr((size_t)ff_p * r.n_used, (size_t)w.ld * (w.f32 ? 4 : 2), 4);
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return with_wpr(wpr, [&](auto n) {
            return check_cuda(launch_k(expert_gate_up_kernel<T, decltype(n)::value>, gv_grid(ff_p, wpr, r.n_used), dim3(GV_WARPS * 32), 0, st,
                                       (const T *)w.w, ff_p, w.ld, (const T *)x, router_logits, r, a, ids, weights, (T *)act),
                              "expert gate/up launch");
        });
    });
}

int32_t launch_expert_down_step(const DenseView &w, uint32_t rows_per_expert, const void *act, const RouterRule &r, const uint32_t *ids,
                                const float *weights, float *y, cudaStream_t st) {
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return check_cuda(launch_k(expert_down_kernel<T>, dim3((rows_per_expert + 1) / 2), dim3(GV_WARPS * 32), 0, st, (const T *)w.w, rows_per_expert, w.ld,
                                   (const T *)act, r.n_used, r.weight_input, ids, weights, y),
                          "expert down launch");
    });
}

}  // namespace cera

// One-column products with dense weights: the decode step's projections, with the work that follows them fused where
// one warp holds all a result needs (the minGRU update, the gated units, the sum over picks).
#include <cooperative_groups.h>

#include "dense_gemv.cuh"
#include "moe_route.cuh"

namespace cera {

namespace {

using namespace gv;

// Rows of GV_LONG vectors and more: where a warp has one to itself, four rows a warp, which share its reads of x, two vectors of each in
// flight, and CTAs of four warps, so that few warps wait for a CTA's last; where warps share it, two rows and four vectors.  Shorter
// rows: one and eight, from 28 rows an SM on two and four.  us, the last / what is chosen: 32768 x 4096 bf16 41.8 / 40.4 (6.6 TB/s), 18560 x 4096
// 26.0 / 24.8, 9600 x 4096 17.6 / 15.7, but with four rows a warp 8192 x 2048 7.7 / 8.7; one row and eight vectors / what is chosen: 4096 x 8192
// 18.1 / 13.5, 4096 x 4096 10.2 / 7.8, but with two rows 3072 x 2048 5.4 / 5.6.
constexpr int GV_LONG_WARPS = 4;
constexpr uint32_t GV_LONG = 512;

// W warps a CTA, WPR of them share R rows, U vectors of each in flight per lane.  What bounds it: HBM.  Of R, W and U the results do
// not depend; WPR fixes the order in which a row is added up, and stays what it is for a shape (see launch_dense_gemv).
template <class T, int W, int R, int WPR, int U>
__global__ void __launch_bounds__(W * 32) gemv_kernel(const T *__restrict__ w, uint32_t rows, uint32_t ld, const T *x, float *y) {
    __shared__ float red[W][R];
    pdl_trigger();
    const int warp = threadIdx.x >> 5;
    const uint32_t g = blockIdx.x * (W / WPR) + warp / WPR;
    RowDot<T, R, U> d;
#pragma unroll
    for (int r = 0; r < R; ++r) d.w[r] = w + (size_t)min(g * R + r, rows - 1) * ld;
    d.start(ld, warp % WPR, WPR);
    d.fetch();
    pdl_wait();
    float acc[R] = {};
    d.run(x, acc);
    group_sum<R, WPR>(acc, red);
    if (warp % WPR == 0 && (threadIdx.x & 31) == 0) {
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

// Rows [0, ff_p) gate, [ff_p, 2 ff_p) up of w; out = unit(gate, up).  W warps a CTA, WPR of them share N units (2 N rows).
template <class T, int W, int N, int WPR, int U>
__global__ void __launch_bounds__(W * 32) gated_unit_step_kernel(const T *__restrict__ w, uint32_t ff_p, uint32_t ld, const T *x, ExpertAct a, T *out) {
    __shared__ float red[W][2 * N];
    pdl_trigger();
    const int warp = threadIdx.x >> 5;
    const uint32_t g = (blockIdx.x * (W / WPR) + warp / WPR) * N;
    RowDot<T, 2 * N, U> d;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        d.w[2 * i] = w + (size_t)min(g + i, ff_p - 1) * ld;
        d.w[2 * i + 1] = d.w[2 * i] + (size_t)ff_p * ld;
    }
    d.start(ld, warp % WPR, WPR);
    d.fetch();
    pdl_wait();
    float acc[2 * N] = {};
    d.run(x, acc);
    group_sum<2 * N, WPR>(acc, red);
    if (warp % WPR == 0 && (threadIdx.x & 31) == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (g + i < ff_p) out[g + i] = Elem<T>::from(gated_unit(acc[2 * i], acc[2 * i + 1], a));
    }
}

// Router logits of one token and the picks, in one launch: a cluster of eight CTAs, eight warps a logit as in the product of its own (which fixes
// the order of its sum), the logits stored into the first CTA's shared memory, which scores and picks.  Every CTA of the experts' gate / up product
// repeated the pick ahead of its weights before: 14.7 us the two launches together at 32 experts of width 2048, 12.8 now.
constexpr uint32_t RP_CLUSTER = 8, RP_WARPS = 32, RP_ROWS = RP_WARPS / 8;
__global__ void __launch_bounds__(RP_WARPS * 32) router_pick_kernel(const float *__restrict__ w, uint32_t ld, const float *x, RouterRule rule, uint32_t *ids,
                                                                    float *weights) {
    __shared__ float red[RP_WARPS][1], probs[MOE_MAX_EXPERTS], wt[MOE_MAX_USED];
    __shared__ uint32_t picked[MOE_MAX_USED];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // the first CTA's shared memory may be written only once it runs
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    pdl_trigger();
    const uint32_t rank = cluster.block_rank(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *first = cluster.map_shared_rank(probs, 0);
    for (uint32_t e0 = 0; e0 < rule.n_expert; e0 += RP_CLUSTER * RP_ROWS) {
        const uint32_t e = e0 + rank * RP_ROWS + warp / 8;
        RowDot<float, 1, 8> d;
        d.w[0] = w + (size_t)min(e, rule.n_expert - 1) * ld;
        d.start(ld, warp % 8, 8);
        d.fetch();
        if (e0 == 0) {
            pdl_wait();
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        float acc[1] = {};
        d.run(x, acc);
        if (e0) __syncthreads();  // the last round's sums have been read
        group_sum<1, 8>(acc, red);
        if (warp % 8 == 0 && lane == 0 && e < rule.n_expert) first[e] = acc[0];
    }
    cluster.sync();
    if (rank || warp) return;
    moe_scores_warp(probs, rule.n_expert, rule.softmax);
    moe_pick(probs, nullptr, rule.n_expert, rule.n_used, rule.renorm, picked, wt);
    if (lane < rule.n_used) {
        ids[lane] = picked[lane];
        weights[lane] = wt[lane];
    }
}

// grid (row groups, picks).
template <class T, int WPR>
__global__ void __launch_bounds__(GV_WARPS * 32) expert_gate_up_kernel(const T *__restrict__ w, uint32_t ff_p, uint32_t ld, const T *x, const uint32_t *ids,
                                                                       const float *weights, int weight_input, ExpertAct a, T *act) {
    __shared__ float red[GV_WARPS][2];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const uint32_t s = blockIdx.y, e = ids[s];
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
        const float sc = weight_input ? weights[s] : 1.0f;
        act[(size_t)s * ff_p + g] = Elem<T>::from(gated_unit(sc * acc[0], sc * acc[1], a));
    }
}

template <class T, int WPR>
__global__ void __launch_bounds__(GV_WARPS * 32) expert_down_kernel(const T *__restrict__ w, uint32_t rows, uint32_t ld, const T *act, uint32_t n_used,
                                                                    int weight_input, const uint32_t *ids, const float *weights, float *y) {
    __shared__ float red[GV_WARPS][1];
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const uint32_t g = blockIdx.x * (GV_WARPS / WPR) + warp / WPR, gi = min(g, rows - 1);
    // the picks' rows are walked as one row of n_used * ld elements, U vectors of it in flight per lane
    constexpr int U = 8;
    const uint32_t nv = ld / Elem<T>::N, all = n_used * nv, step = 32u * WPR;
    float total[1] = {0.0f};
    for (uint32_t c = (warp % WPR) * 32u + (threadIdx.x & 31); c < all; c += U * step) {
        uint4 wb[U], xb[U];
        float sc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t v = c + u * step, s = v / nv;
            if (v < all) {
                wb[u] = ld_stream(reinterpret_cast<const uint4 *>(w + ((size_t)ids[s] * rows + gi) * ld) + (v - s * nv));
                xb[u] = *(reinterpret_cast<const uint4 *>(act) + v);
                sc[u] = weight_input ? 1.0f : weights[s];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c + u * step < all) {
                float wf[Elem<T>::N], xf[Elem<T>::N], a = 0.0f;
                Elem<T>::unpack(wb[u], wf);
                Elem<T>::unpack(xb[u], xf);
#pragma unroll
                for (int i = 0; i < Elem<T>::N; ++i) a = fmaf(wf[i], xf[i], a);
                total[0] = fmaf(sc[u], a, total[0]);
            }
    }
    group_sum<1, WPR>(total, red);
    if (warp % WPR == 0 && (threadIdx.x & 31) == 0 && g < rows) y[g] = total[0];
}

}  // namespace

// The warps that share a row (wpr) are part of the result: they fix the order of its additions, and with it each last bit, which the
// rounding to bf16 widens and a router with two experts almost level turns into another pick.  A shape keeps its wpr; only the layout
// around it is free.
int32_t launch_dense_gemv(const DenseView &w, const void *x, float *y, cudaStream_t st) {
    const bool pairs = w.rows >= (uint32_t)sm_count() * 28;
    const int wpr = pick_wpr(pairs ? (w.rows + 1) / 2 : w.rows, (size_t)w.ld * (w.f32 ? 4 : 2), pairs ? 4 : 8);
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        const bool long_rows = w.ld / Elem<T>::N >= GV_LONG;
        if (wpr == 1 && long_rows)
            return check_cuda(launch_k(gemv_kernel<T, GV_LONG_WARPS, 4, 1, 2>, gv_grid((w.rows + 3) / 4, 1, 1, GV_LONG_WARPS), dim3(GV_LONG_WARPS * 32), 0, st,
                                       (const T *)w.w, w.rows, w.ld, (const T *)x, y),
                              "dense gemv launch");
        return with_wpr(wpr, [&](auto n) {
            constexpr int WPR = decltype(n)::value, R = WPR == 8 ? 1 : 2;  // (eight warps share a row where there are few: a CTA each)
            if (R == 2 && (pairs || long_rows))
                return check_cuda(launch_k(gemv_kernel<T, GV_WARPS, R, WPR, 8 / R>, gv_grid((w.rows + R - 1) / R, wpr), dim3(GV_WARPS * 32), 0, st,
                                           (const T *)w.w, w.rows, w.ld, (const T *)x, y),
                                  "dense gemv launch");
            return check_cuda(launch_k(gemv_kernel<T, GV_WARPS, 1, WPR, 8>, gv_grid(w.rows, wpr), dim3(GV_WARPS * 32), 0, st, (const T *)w.w, w.rows, w.ld,
                                       (const T *)x, y),
                              "dense gemv launch");
        });
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
    const int wpr = pick_wpr(ff_p, (size_t)w.ld * (w.f32 ? 4 : 2), 4);
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        if (wpr == 1 && w.ld / Elem<T>::N >= GV_LONG)
            return check_cuda(launch_k(gated_unit_step_kernel<T, GV_LONG_WARPS, 2, 1, 2>, gv_grid((ff_p + 1) / 2, 1, 1, GV_LONG_WARPS),
                                       dim3(GV_LONG_WARPS * 32), 0, st, (const T *)w.w, ff_p, w.ld, (const T *)x, a, (T *)out),
                              "gated unit launch");
        return with_wpr(wpr, [&](auto n) {
            return check_cuda(launch_k(gated_unit_step_kernel<T, GV_WARPS, 1, decltype(n)::value, 4>, gv_grid(ff_p, wpr), dim3(GV_WARPS * 32), 0, st,
                                       (const T *)w.w, ff_p, w.ld, (const T *)x, a, (T *)out),
                              "gated unit launch");
        });
    });
}

int32_t launch_router_pick_step(const DenseView &router, const float *x, const RouterRule &r, uint32_t *ids, float *weights, cudaStream_t st) {
    if (!router.f32 || r.n_expert == 0 || r.n_expert > MOE_MAX_EXPERTS || r.n_used == 0 || r.n_used > MOE_MAX_USED || r.n_used > r.n_expert)
        return fail(CERA_CUDA_ERR_BAD_ARG, "router: %u experts, %u used (limits %d, %d)", r.n_expert, r.n_used, MOE_MAX_EXPERTS, MOE_MAX_USED);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(RP_CLUSTER);
    cfg.blockDim = dim3(RP_WARPS * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = RP_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch();
    return check_cuda(cudaLaunchKernelEx(&cfg, router_pick_kernel, (const float *)router.w, router.ld, x, r, ids, weights), "router launch");
}

int32_t launch_expert_gate_up_step(const DenseView &w, const void *x, const uint32_t *ids, const float *weights, const RouterRule &r, uint32_t ff_p,
                                   const ExpertAct &a, void *act, cudaStream_t st) {
    const int wpr = pick_wpr((size_t)ff_p * r.n_used, (size_t)w.ld * (w.f32 ? 4 : 2), 4);
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return with_wpr(wpr, [&](auto n) {
            return check_cuda(launch_k(expert_gate_up_kernel<T, decltype(n)::value>, gv_grid(ff_p, wpr, r.n_used), dim3(GV_WARPS * 32), 0, st,
                                       (const T *)w.w, ff_p, w.ld, (const T *)x, ids, weights, r.weight_input, a, (T *)act),
                              "expert gate/up launch");
        });
    });
}

int32_t launch_expert_down_step(const DenseView &w, uint32_t rows_per_expert, const void *act, const RouterRule &r, const uint32_t *ids,
                                const float *weights, float *y, cudaStream_t st) {
    const int wpr = pick_wpr(rows_per_expert, (size_t)w.ld * (w.f32 ? 4 : 2), 2);
    count_launch();
    return with_type(w.f32, [&](auto t) {
        using T = decltype(t);
        return with_wpr(wpr, [&](auto n) {
            return check_cuda(launch_k(expert_down_kernel<T, decltype(n)::value>, gv_grid(rows_per_expert, wpr), dim3(GV_WARPS * 32), 0, st,
                                       (const T *)w.w, rows_per_expert, w.ld, (const T *)act, r.n_used, r.weight_input, ids, weights, y),
                              "expert down launch");
        });
    });
}

}  // namespace cera

// Routed feed-forward of ONE token, the decode step of a mixture-of-experts model, in three launches (moe.cu: batches and expert parallelism).
//
// What bounds it is latency: 16.5 MB of Q4_0 (four experts of 2048 x 1792) are 2.6 us of HBM, and the batch form's ten launches in a row took 39 us
// on the device, most of them a few dependent round trips each.  Here
//   moe_token_route_kernel  a cluster of eight CTAs: a warp per expert's score, the token's Q8_0 blocks beside them; the scores meet in the
//                           first CTA's shared memory, which picks and writes ids and weights, the caller's copies included.
//   moe_token_up_kernel     a CTA per 32 units of a picked expert: gate and up rows, silu(gate) up, and the Q8_0 block they are.
//   moe_token_down_kernel   a warp per output: its row of every picked expert, added up in pick order.
// Every sum is formed as the batch form forms it for one token, bit for bit.
// 32 experts, 4 used, 2048 x 1792, Q4_0: 45 us a call before, 19.4 now, call after call; a call by itself is 20.0 us on the device, from one kernel's end to
// the next one's 5.9 + 8.3 + 5.8.
#include <cooperative_groups.h>

#include "gemv_item.cuh"
#include "moe_route.cuh"

namespace cera {

namespace {

namespace cg = cooperative_groups;

constexpr uint32_t MT_CLUSTER = 8, MT_WARPS = 8, MT_THREADS = MT_WARPS * 32, MT_UP_WARPS = 16;
constexpr int MT_AHEAD = 16;  // vectors of a router row that a lane requests before the token is there

__global__ void __launch_bounds__(MT_THREADS) moe_token_route_kernel(const float *__restrict__ x, const float *__restrict__ router, const float *__restrict__ bias,
                                                                     uint32_t hidden, uint32_t n_expert, uint32_t n_used, int softmax_gate, float *scales,
                                                                     int8_t *quants, int16_t *sums, uint32_t *ids, float *weights, uint32_t *ids_out,
                                                                     float *weights_out) {
    __shared__ float probs[MOE_MAX_EXPERTS];
    __shared__ uint32_t picked[MOE_MAX_USED];
    __shared__ float w[MOE_MAX_USED];
    cg::cluster_group cluster = cg::this_cluster();
    // the first CTA's shared memory may be written only once it runs: everybody arrives here and waits just before the stores
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    pdl_trigger();
    const uint32_t rank = cluster.block_rank(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, all = MT_CLUSTER * MT_THREADS, nv = hidden / 4;
    uint32_t e = rank * MT_WARPS + warp;
    float4 ahead[MT_AHEAD];
#pragma unroll
    for (int i = 0; i < MT_AHEAD; ++i)
        if (e < n_expert && lane + 32 * i < nv) ahead[i] = __ldg(reinterpret_cast<const float4 *>(router + (size_t)e * hidden) + lane + 32 * i);
    pdl_wait();
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    float *first = cluster.map_shared_rank(probs, 0);
    bool ready = false;
    for (; e < n_expert; e += MT_CLUSTER * MT_WARPS) {
        const float4 *r = reinterpret_cast<const float4 *>(router + (size_t)e * hidden);
        float acc = 0.0f;
        auto add = [&](const float4 &rv, const float4 &xv) { acc = fmaf(rv.w, xv.w, fmaf(rv.z, xv.z, fmaf(rv.y, xv.y, fmaf(rv.x, xv.x, acc)))); };
        uint32_t i = lane;
        if (!ready) {
#pragma unroll
            for (int j = 0; j < MT_AHEAD; ++j)
                if (lane + 32 * j < nv) add(ahead[j], x4[lane + 32 * j]);
            i += 32 * MT_AHEAD;
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            ready = true;
        }
#pragma unroll 8
        for (; i < nv; i += 32) add(__ldg(r + i), x4[i]);
        acc = warp_sum(acc);
        if (lane == 0) first[e] = acc;
    }
    if (!ready) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    for (uint32_t v0 = 0; v0 < nv; v0 += all) {  // nv is a multiple of 8: a block's eight lanes are all in or all out
        const uint32_t v = v0 + rank * MT_THREADS + threadIdx.x;
        const bool in = v < nv;
        const float4 a = in ? x4[v] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float q[4] = {a.x, a.y, a.z, a.w};
        const QuantQuad o = quantize_quad(q);
        if (in) {
            reinterpret_cast<uint32_t *>(quants)[v] = o.quants;
            if ((lane & 7) == 0) scales[v >> 3] = o.scale;
            if ((lane & 3) == 0) sums[v >> 2] = (int16_t)o.half_sum;
        }
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // every score is there
    if (rank || warp) return;
    moe_scores_warp(probs, n_expert, softmax_gate);
    moe_pick(probs, bias, n_expert, n_used, 1, picked, w);
    if (lane < n_used) {
        ids[lane] = picked[lane];
        weights[lane] = w[lane];
        if (ids_out) ids_out[lane] = picked[lane];
        if (weights_out) weights_out[lane] = w[lane];
    }
}

// grid (ff / 32, picks).  A warp has two units, four rows: their loads, of up to two items a lane, are under way together.
template <int T>
__global__ void __launch_bounds__(MT_UP_WARPS * 32) moe_token_up_kernel(const WeightView gate, const WeightView up, uint32_t hidden, uint32_t ff, const ActView x,
                                                                        const uint32_t *__restrict__ ids, float *scales, int8_t *quants, int16_t *sums) {
    using F = Fmt<T>;
    constexpr int R = 32 / MT_UP_WARPS, AHEAD = T == CERA_TYPE_Q4_0 || T == CERA_TYPE_Q4_1 || T == CERA_TYPE_Q8_0 ? 2 : 1;  // (K-quants: registers)
    __shared__ float s_of[2][32];  // gate, up
    pdl_trigger();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pick = blockIdx.y, items = hidden >> 5;
    const size_t row0 = (size_t)ids[pick] * ff + blockIdx.x * 32 + warp * R;
    float acc[2][R][1] = {};
    for (uint32_t item0 = lane; item0 < items; item0 += 32 * AHEAD) {
        typename F::Raw raw[AHEAD][2][R];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (item0 + 32 * a < items) {
                    raw[a][0][i] = F::load(gate, row0 + i, (int)(item0 + 32 * a));
                    raw[a][1][i] = F::load(up, row0 + i, (int)(item0 + 32 * a));
                }
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
            if (item0 + 32 * a < items)
#pragma unroll
                for (int i = 0; i < R; ++i)
#pragma unroll
                    for (int m = 0; m < 2; ++m) accumulate_item<T, 1>(raw[a][m][i], (int)(item0 + 32 * a), x, hidden, acc[m][i]);
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const float v = warp_sum(acc[m][i][0]);
            if (lane == 0) s_of[m][warp * R + i] = v;
        }
    __syncthreads();
    if (warp) return;
    float scale;
    int hs;
    const int q = quantize_lane(silu_mul(s_of[0][lane], s_of[1][lane]), scale, hs);
    const size_t b = (size_t)pick * (ff / 32) + blockIdx.x;
    quants[b * 32 + lane] = (int8_t)q;
    if (lane == 0) scales[b] = scale;
    if ((lane & 15) == 0) sums[b * 2 + (lane >> 4)] = (int16_t)hs;
}

// grid ceil(hidden / MT_WARPS).  Multiply and add rounded separately, in pick order, as the batch's combination.
template <int T>
__global__ void __launch_bounds__(MT_THREADS) moe_token_down_kernel(const WeightView down, uint32_t hidden, uint32_t ff, uint32_t n_used, const ActView x,
                                                                    const uint32_t *__restrict__ ids, const float *__restrict__ weights, float *__restrict__ out) {
    using F = Fmt<T>;
    constexpr int R = 4;
    pdl_trigger();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31, row = blockIdx.x * MT_WARPS + (threadIdx.x >> 5);
    if (row >= hidden) return;
    const uint32_t items = ff >> 5;
    float sum = 0.0f;
    for (uint32_t s0 = 0; s0 < n_used; s0 += R) {
        float acc[R][1] = {};
        size_t wrow[R];
#pragma unroll
        for (uint32_t s = 0; s < R; ++s) wrow[s] = (size_t)ids[min(s0 + s, n_used - 1)] * hidden + row;
        for (uint32_t item = lane; item < items; item += 32) {
            typename F::Raw raw[R];
#pragma unroll
            for (uint32_t s = 0; s < R; ++s) raw[s] = F::load(down, wrow[s], (int)item);
#pragma unroll
            for (uint32_t s = 0; s < R; ++s) {
                const size_t e = min(s0 + s, n_used - 1);
                accumulate_item<T, 1>(raw[s], (int)item, ActView{x.scales + e * (ff / 32), x.quants + e * ff, x.sums + e * (ff / 16)}, ff, acc[s]);
            }
        }
#pragma unroll
        for (uint32_t s = 0; s < R; ++s) {
            const float v = warp_sum(acc[s][0]);
            if (s0 + s < n_used) sum = __fadd_rn(sum, __fmul_rn(weights[s0 + s], v));
        }
    }
    if (lane == 0) out[row] = sum;
}

}  // namespace

int32_t launch_moe_token(const MoeToken &p, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(MT_CLUSTER);
    cfg.blockDim = dim3(MT_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = MT_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch(3);
    CERA_TRY(check_cuda(cudaLaunchKernelEx(&cfg, moe_token_route_kernel, p.x, p.router, p.bias, p.hidden, p.n_expert, p.n_used, p.softmax_gate, p.in.scales,
                                           p.in.quants, p.in.sums, p.ids, p.weights, p.ids_out, p.weights_out),
                        "moe (one token) route launch"));
    const ActView in{p.in.scales, p.in.quants, p.in.sums}, mid{p.mid.scales, p.mid.quants, p.mid.sums};
    CERA_DISPATCH_BLOCK_TYPE(
        p.gate.type,
        CERA_TRY(check_cuda(launch_k(moe_token_up_kernel<TT>, dim3(p.ff / 32, p.n_used), dim3(MT_UP_WARPS * 32), 0, st, p.gate, p.up, p.hidden, p.ff, in,
                                     (const uint32_t *)p.ids, p.mid.scales, p.mid.quants, p.mid.sums),
                            "moe (one token) gate / up launch"));
        return check_cuda(launch_k(moe_token_down_kernel<TT>, dim3((p.hidden + MT_WARPS - 1) / MT_WARPS), dim3(MT_THREADS), 0, st, p.down, p.hidden, p.ff, p.n_used,
                                   mid, (const uint32_t *)p.ids, (const float *)p.weights, p.out),
                          "moe (one token) down launch"));
    return CERA_CUDA_OK;
}

}  // namespace cera

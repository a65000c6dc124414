// Decode attention in the reference's own arithmetic order, so that its output is bit-identical to
// what cera computes on an x86 host with AVX2+FMA (cera/src/model/transformer.rs:1166-1305 calling
// cera/src/backend/cpu.rs:3522-3625 and softmax_inplace, cpu.rs:2617-2633), for head sizes that are a
// multiple of 32 up to 256 and up to 8 query heads per KV head.
//
// The reference computes, per query head: every score as two 8-lane FMA accumulators over alternating
// 8-wide slices of the head (16 chains of head_dim/16 FMAs), added lane-wise, reduced in the hsum256
// order and multiplied by the scale; then a plain softmax over ALL positions (maximum, ggml_expf,
// f64 sum, one multiplication by (float)(1/sum)); then out[d] = fma(p[t], V[t][d], out[d]) for t in
// position order.  The last step is a serial chain per output element that an online-softmax
// (flash-decode) kernel cannot reproduce, so the work is split differently here:
//
//   scores  : sixteen positions per warp, two lanes per position: lane bit 0 picks the accumulator (a), a lane holds its
//             eight chains, so a K row arrives in 128-bit loads and is read once for all heads of the group; five shuffles
//             add the chains in the reference's order.
//   up to 1024 positions and heads of 64, 128 or 256, ONE launch (attn_fused_exact_kernel): the hd / 32 CTAs of a KV head are a cluster, each scores a
//             share of the positions into the tables of all, then runs the softmax and the value chains of its 32 dims.
//   beyond  : attn_scores_exact_kernel writes scores and the maximum of every sixteen; attn_exp_exact_kernel turns them into
//             exponentials in place and leaves one f64 sum per 1024 positions; attn_chain_exact_kernel multiplies by
//             1 / sum and walks the chains, one warp per (head, 32 dims), fed by copying warps through a ring.
//
// The chain of an output element is one dependent FMA per position, 4 cycles: 2.1 ns per position at 1.96 GHz bounds a long
// context (34 us at 16384).  What a chain warp adds to that is the issue of its loads, which do not overlap the FMAs they stand
// between, and the wait for them when other warps keep the load / store unit busy: V therefore arrives by TMA, probabilities
// are multiplied by 1 / sum beforehand and fetched four at a time, and values four or eight positions a load, 32 positions ahead of
// their FMAs.  Alone on an SM: 5.1 cycles per position (f32; f16 6.0), 6.5 and 6.7 with a load per position, 10.8 eight positions
// ahead; V transposed to [dim][position] by copying warps - 5.1 alone - costs 9 to 13 beside those warps.
//
// The f64 sum of the exponentials is a tree, the reference's a left-to-right loop: the two can differ
// in the last bits of the f64 sum, which survive the narrowing to f32 only in about one softmax in
// 10^7 (and not at all while every partial sum is exactly representable, which holds whenever the
// probabilities span fewer than ~29 binary orders of magnitude).
#include <cooperative_groups.h>

#include <cstdlib>
#include <cstring>

#include "act.cuh"
#include "ops.h"
#include "tensor_map.h"
#include "tma.cuh"

namespace cg = cooperative_groups;

namespace cera {

namespace {

constexpr int AX_VTHREADS = 512;   // threads of the fused kernel

__device__ unsigned int g_ax_status = 0;  // bit 0: a chain warp's wait ran out, bit 1: a copying warp's

// This lane's half (accumulator a) of one K row: chunks 2j + a of eight elements, j = 0 .. HD/16 - 1.  `vec`: the cache starts
// on a 16-byte boundary (every row and chunk then does).
template <int HD, bool F16>
__device__ __forceinline__ void ax_load_k(float (&k)[HD / 16][8], const void *__restrict__ kc, size_t row, uint32_t a, bool vec) {
    const size_t e0 = row + 8 * a;
    if (vec) {
        if constexpr (F16) {
            uint4 raw[HD / 16];
#pragma unroll
            for (int j = 0; j < HD / 16; ++j) raw[j] = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(kc) + e0 + 16 * j));
#pragma unroll
            for (int j = 0; j < HD / 16; ++j) {
                const uint32_t w[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    k[j][2 * i] = h2f((uint16_t)(w[i] & 0xFFFF));
                    k[j][2 * i + 1] = h2f((uint16_t)(w[i] >> 16));
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < HD / 16; ++j) {
                const float4 *src = reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(kc) + e0 + 16 * j);
                const float4 lo = __ldg(src), hi = __ldg(src + 1);
                k[j][0] = lo.x, k[j][1] = lo.y, k[j][2] = lo.z, k[j][3] = lo.w;
                k[j][4] = hi.x, k[j][5] = hi.y, k[j][6] = hi.z, k[j][7] = hi.w;
            }
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < HD / 16; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            k[j][i] = F16 ? __half2float(__ldg(reinterpret_cast<const __half *>(kc) + e0 + 16 * j + i)) : __ldg(reinterpret_cast<const float *>(kc) + e0 + 16 * j + i);
}

// Scaled score of one head (qh: its query in shared memory) against the row whose halves this lane and lane ^ X hold; both
// lanes return it.  Chain (a, i) multiplies elements 16j + 8a + i in the order of j; then the two accumulators are added lane by
// lane and reduced as hsum256 does: i and i + 4, then (0,2) and (1,3), then the two.
template <int HD, int X>
__device__ __forceinline__ float ax_score(const float *qh, const float (&k)[HD / 16][8], uint32_t a, float scale) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll
    for (int j = 0; j < HD / 16; ++j) {
        const float4 lo = *reinterpret_cast<const float4 *>(qh + 16 * j + 8 * a), hi = *reinterpret_cast<const float4 *>(qh + 16 * j + 8 * a + 4);
        acc[0] = fmaf(lo.x, k[j][0], acc[0]);
        acc[1] = fmaf(lo.y, k[j][1], acc[1]);
        acc[2] = fmaf(lo.z, k[j][2], acc[2]);
        acc[3] = fmaf(lo.w, k[j][3], acc[3]);
        acc[4] = fmaf(hi.x, k[j][4], acc[4]);
        acc[5] = fmaf(hi.y, k[j][5], acc[5]);
        acc[6] = fmaf(hi.z, k[j][6], acc[6]);
        acc[7] = fmaf(hi.w, k[j][7], acc[7]);
    }
    float r[4];  // both accumulators' lanes a, a + 2, a + 4, a + 6
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const float keep = a ? acc[2 * m + 1] : acc[2 * m], send = a ? acc[2 * m] : acc[2 * m + 1];
        r[m] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, X));
    }
    const float u = __fadd_rn(__fadd_rn(r[0], r[2]), __fadd_rn(r[1], r[3]));
    return __fmul_rn(__fadd_rn(u, __shfl_xor_sync(0xffffffffu, u, X)), scale);
}

// Scores of all heads of one KV head, and the maximum of every sixteen positions.  grid (any, n_kv), AX_SWARPS warps;
// dynamic shared memory: G * HD floats of q.  ws: scores [n_heads][ld]; aux: [n_heads][ld], its first ld / 16 entries per head
// receive the maxima.  16384 f16 positions, 32 heads of 128 in groups of 4: 33.5 MB of keys in 15.7 us (36 us with a half-warp
// per position and head, whose 2-byte loads left 8 KB in flight per SM).
constexpr int AX_SWARPS = 8;
template <int HD, bool F16>
__global__ void __launch_bounds__(AX_SWARPS * 32)
attn_scores_exact_kernel(const float *__restrict__ q, const void *__restrict__ kc, int vec, uint32_t seq_len,
                         const uint32_t *__restrict__ seq_dev, uint32_t n_kv, uint32_t G, float scale, float *__restrict__ ws,
                         float *__restrict__ aux, uint32_t ld) {
    extern __shared__ __align__(16) float ax_q[];
    pdl_trigger();
    pdl_wait();
    const uint32_t seq = seq_dev ? min(*seq_dev, ld) : seq_len;
    const uint32_t kvh = blockIdx.y;
    for (uint32_t i = threadIdx.x; i < G * HD; i += blockDim.x) ax_q[i] = q[(size_t)kvh * G * HD + i];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, a = lane & 1;
    const size_t kv_dim = (size_t)n_kv * HD;
    const uint32_t tiles = (seq + 15) / 16;
    for (uint32_t tile = blockIdx.x * AX_SWARPS + warp; tile < tiles; tile += gridDim.x * AX_SWARPS) {
        const uint32_t t = tile * 16 + (lane >> 1);
        float k[HD / 16][8];
        ax_load_k<HD, F16>(k, kc, (size_t)min(t, seq - 1) * kv_dim + (size_t)kvh * HD, a, vec);
        for (uint32_t h = 0; h < G; ++h) {
            const float s = ax_score<HD, 1>(ax_q + h * HD, k, a, scale);
            const size_t row = (size_t)(kvh * G + h) * ld;
            if (a == 0 && t < seq) ws[row + t] = s;
            float mx = t < seq ? fmaxf(-INFINITY, s) : -INFINITY;  // f32::max fold: NaN scores are ignored
#pragma unroll
            for (int o = 16; o > 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0) aux[row + tile] = mx;
        }
    }
}

// Exponentials of one head's scores, in place, and their f64 sum per AX_EPOS positions (thread-strided partials, xor shuffles,
// warps in index order) behind the maxima in aux.  grid (any, n_heads), AX_ETHREADS threads.
constexpr uint32_t AX_EPOS = 1024, AX_ETHREADS = 256;
__device__ __host__ __forceinline__ uint32_t ax_sums_at(uint32_t ld) { return ld / 16; }  // 2 * ceil(ld / 1024) words follow: within ld, a multiple of 64
__global__ void __launch_bounds__(AX_ETHREADS)
attn_exp_exact_kernel(float *__restrict__ ws, float *__restrict__ aux, uint32_t ld, uint32_t seq_len, const uint32_t *__restrict__ seq_dev) {
    __shared__ float red_f[AX_ETHREADS / 32];
    __shared__ double red_d[AX_ETHREADS / 32];
    pdl_trigger();
    pdl_wait();
    const uint32_t seq = seq_dev ? min(*seq_dev, ld) : seq_len;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x * AX_EPOS >= seq) return;
    float *row = ws + (size_t)blockIdx.y * ld;
    float *maxima = aux + (size_t)blockIdx.y * ld;
    float mx = -INFINITY;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < (seq + 15) / 16; i += AX_ETHREADS) mx = fmaxf(mx, maxima[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red_f[warp] = mx;
    __syncthreads();
    mx = red_f[0];
#pragma unroll
    for (uint32_t w = 1; w < AX_ETHREADS / 32; ++w) mx = fmaxf(mx, red_f[w]);
    for (uint32_t part = blockIdx.x; part * AX_EPOS < seq; part += gridDim.x) {
        double sum = 0.0;
#pragma unroll
        for (uint32_t i = 0; i < AX_EPOS / AX_ETHREADS; ++i) {
            const uint32_t t = part * AX_EPOS + i * AX_ETHREADS + threadIdx.x;
            if (t < seq) {
                const float e = ggml_expf(__fsub_rn(row[t], mx));
                row[t] = e;
                sum += (double)e;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) red_d[warp] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t w = 1; w < AX_ETHREADS / 32; ++w) sum += red_d[w];
            // two words: the workspace is only known to be aligned to floats
            float *dst = maxima + ax_sums_at(ld) + 2 * part;
            dst[0] = __int_as_float(__double2hiint(sum));
            dst[1] = __int_as_float(__double2loint(sum));
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void ax_cp16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tma::smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void ax_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ax_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Which of a slice's 32 dims a lane's chain is, and a warp's chains in the order of the dims.
template <bool F16>
__device__ __forceinline__ uint32_t ax_dim(uint32_t lane) { return F16 ? lane % 4 * 8 + lane / 4 : lane; }
template <bool F16>
__device__ __forceinline__ float ax_by_dim(float acc, uint32_t lane) { return F16 ? __shfl_sync(0xffffffffu, acc, lane % 8 * 4 + lane / 8) : acc; }

// cnt positions of one lane's chain: out = fma(p, V, out) in position order.  v: the first of cnt rows of 32 dims; pa: the head's
// probabilities (shared-memory addresses, 16-byte aligned).  Values come by ldmatrix, whose eight 16-byte rows may lie anywhere: f32, a
// row of 32 dims is one 8 x 8 matrix of 32-bit words, word l of it lane l's; f16, the four pieces of two rows in turn, transposed, are
// lane (g, j)'s dim 8 j + g of both.  So one load brings four positions (f16: eight), where one load per position cost the chain 7.9 cycles
// beside the TMA thread.  The loads are volatile so that the compiler leaves them 32 positions ahead of their FMAs.
template <bool F16>
__device__ __forceinline__ float ax_chain(uint32_t v, uint32_t pa, uint32_t cnt, float acc) {
    constexpr int R = 8, ROW = F16 ? 64 : 128, PER = F16 ? 2 : 1, N = R / PER;  // quads of positions in registers; of a load; loads
    const uint32_t lane = threadIdx.x & 31;
    // the matrix row whose address this lane gives: position, piece
    const uint32_t at = F16 ? (lane >> 3) * 2 + (lane & 1) : lane >> 3, piece = F16 ? (lane >> 1) & 3 : lane & 7;
    uint32_t va = v + at * ROW + piece * 16;
    auto ld_v = [](uint32_t (&r)[4], uint32_t a) {
        if constexpr (F16)
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
        else
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    };
    auto ld_p = [](float4 &r, uint32_t a) {
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(a) : "memory");
    };
    // four positions, the q-th quad of a load
    auto quad = [&](const uint32_t (&r)[4], int q, const float4 &p) {
        if constexpr (F16) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&r[2 * q])), b = __half22float2(*reinterpret_cast<const __half2 *>(&r[2 * q + 1]));
            acc = fmaf(p.w, b.y, fmaf(p.z, b.x, fmaf(p.y, a.y, fmaf(p.x, a.x, acc))));
        } else {
            acc = fmaf(p.w, __uint_as_float(r[3]), fmaf(p.z, __uint_as_float(r[2]), fmaf(p.y, __uint_as_float(r[1]), fmaf(p.x, __uint_as_float(r[0]), acc))));
        }
    };
    const uint32_t full = cnt / (4 * R);
    if (full) {
        uint32_t x[N][4];
        float4 p[R];
#pragma unroll
        for (int i = 0; i < N; ++i) ld_v(x[i], va + i * 4 * PER * ROW);
#pragma unroll
        for (int i = 0; i < R; ++i) ld_p(p[i], pa + 16 * i);
#pragma unroll 1
        for (uint32_t b = 1; b < full; ++b) {
            va += 4 * R * ROW;
            pa += 16 * R;
#pragma unroll
            for (int i = 0; i < N; ++i) {
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    quad(x[i], q, p[i * PER + q]);
                    ld_p(p[i * PER + q], pa + 16 * (i * PER + q));
                }
                ld_v(x[i], va + i * 4 * PER * ROW);
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) quad(x[i / PER], i % PER, p[i]);
        pa += 16 * R;
    }
    // the rest one by one
    const uint32_t done = full * 4 * R, el = v + ax_dim<F16>(lane) * (F16 ? 2 : 4);
#pragma unroll 4
    for (uint32_t i = done; i < cnt; ++i, pa += 4) {
        uint32_t x, p;
        if constexpr (F16) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(x) : "r"(el + i * ROW) : "memory");
        else asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(el + i * ROW) : "memory");
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(p) : "r"(pa) : "memory");
        acc = fmaf(__uint_as_float(p), F16 ? h2f((uint16_t)x) : __uint_as_float(x), acc);
    }
    return acc;
}

// One warp writes the 32 outputs of a head's block: f32 (o: this lane's index) and, if asked for, Q8_0.
__device__ __forceinline__ void ax_emit(float acc, size_t o, uint32_t d, float *__restrict__ out, float *scales, int8_t *quants, int16_t *sums,
                                        const TpHook &tp) {
    out[o] = acc;
    if (quants) {
        // Q8_0 of the 32-dim block this warp holds (cera/src/backend/cpu.rs:942-958)
        const float av = fabsf(acc);
        float amax = av == av ? av : 0.0f;
#pragma unroll
        for (int sft = 16; sft > 0; sft >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, sft));
        const float dd = __fdiv_rn(amax, 127.0f);
        const float r = __fdiv_rn(1.0f, dd);
        const float id = (dd != 0.0f && isfinite(r)) ? r : 0.0f;
        const float pq = rintf(__fmul_rn(acc, id));
        const int qv = pq != pq ? 0 : (int)fminf(fmaxf(pq, -128.0f), 127.0f);
        int s16 = qv;  // sums of the two 16-element halves
#pragma unroll
        for (int sft = 8; sft > 0; sft >>= 1) s16 += __shfl_xor_sync(0xffffffffu, s16, sft);
        const float sc = __half2float(__float2half_rn(dd));
        quants[o] = (int8_t)qv;
        if (d == 0) scales[o / 32] = sc;
        if ((d & 15) == 0) sums[o / 16] = (int16_t)s16;
        if (tp.push) {
            // peers receive whole 32-bit words: lanes 0, 4, 8, ... gather their four quants
            uint32_t packed = (uint32_t)(uint8_t)qv;
            packed |= (uint32_t)(uint8_t)__shfl_down_sync(0xffffffffu, qv, 1) << 8;
            packed |= (uint32_t)(uint8_t)__shfl_down_sync(0xffffffffu, qv, 2) << 16;
            packed |= (uint32_t)(uint8_t)__shfl_down_sync(0xffffffffu, qv, 3) << 24;
            if ((d & 3) == 0) tp_push(tp.ctx, reinterpret_cast<uint32_t *>(quants + o), packed);
            if (d == 0) tp_push(tp.ctx, scales + o / 32, sc);
            if ((d & 15) == 0) tp_push(tp.ctx, sums + o / 16, (int16_t)s16);
        }
    }
}

// The value chains of a long context.  grid (hd / 32, n_kv, ceil(G / AXC_HEADS)); a CTA has one warp per head of its share, one
// thread that requests V tiles (AXC_T positions x 32 dims, two TMA boxes) and three warps that prepare the heads' probabilities
// of every third tile.  Slots of the ring are handed over through mbarriers, every wait bounded.  The positions of a last,
// incomplete box are copied by the probability warp: a box may not reach past the cache.  Two heads per CTA: one would read
// every V slice from L2 once per head, four would share one load / store unit among four chains.
// 16384 f16 positions, 32 heads of 128 in groups of 4: 57.6 us, and 77 us with the two kernels ahead.
constexpr int AXC_HEADS = 2, AXC_PWARPS = 3, AXC_T = 512, AXC_BOX = 256;
constexpr uint32_t AXC_THREADS = (AXC_HEADS + AXC_PWARPS + 1) * 32;
template <bool F16>
struct AxChain {
    static constexpr int STAGES = F16 ? 4 : 3;
    // a probability warp waits for the slot of its next tile by parity: the phase before that one must be over, which the tile it
    // filled last shows only while it skips no more tiles than there are slots
    static_assert(AXC_PWARPS <= STAGES, "a parity wait may not run two phases ahead");
    static constexpr uint32_t ROW = 32 * (F16 ? 2 : 4), V_BYTES = AXC_T * ROW, STAGE = V_BYTES + AXC_HEADS * AXC_T * 4, SMEM = STAGES * STAGE + 128;
};
template <bool F16>
__global__ void __launch_bounds__(AXC_THREADS)
attn_chain_exact_kernel(const __grid_constant__ CUtensorMap v_map, const float *__restrict__ ws, const float *__restrict__ aux, uint32_t ld,
                        const void *__restrict__ vc, uint32_t seq_len, const uint32_t *__restrict__ seq_dev, uint32_t n_kv, uint32_t G, uint32_t hd,
                        float *__restrict__ out, float *scales, int8_t *quants, int16_t *sums, const TpHook tp) {
    using C = AxChain<F16>;
    extern __shared__ __align__(128) char axc_dyn[];
    __shared__ uint64_t full[C::STAGES], empty[C::STAGES];
    __shared__ uint32_t gave_up;
    char *ring = axc_dyn + ((128 - (tma::smem_u32(axc_dyn) & 127)) & 127);
    const uint32_t kvh = blockIdx.y, d0 = blockIdx.x * 32, h0 = blockIdx.z * AXC_HEADS, nh = min((uint32_t)AXC_HEADS, G - h0);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int i = 0; i < C::STAGES; ++i) {
            tma::mbar_init(full + i, 2);    // the V request's expect_tx, the probability warp
            tma::mbar_init(empty + i, nh);  // the chain warps
        }
        tma::mbar_init_fence();
    }
    __syncthreads();
    pdl_trigger();
    pdl_wait();
    const uint32_t seq = seq_dev ? min(*seq_dev, ld) : seq_len;
    const uint32_t n_tiles = (seq + AXC_T - 1) / AXC_T;
    if (warp == AXC_HEADS + AXC_PWARPS) {
        if (lane) return;
        uint32_t tile = 0;
        for (; tile < n_tiles; ++tile) {
            const uint32_t slot = tile % C::STAGES;
            if (tile >= C::STAGES && !tma::mbar_wait_blocking(empty + slot, (tile / C::STAGES - 1) & 1, &gave_up, &g_ax_status, 2u)) break;
            const uint32_t boxes = min((uint32_t)AXC_T, seq - tile * AXC_T) / AXC_BOX;
            if (!boxes) {
                tma::mbar_arrive(full + slot);
                continue;
            }
            tma::mbar_expect_tx(full + slot, boxes * AXC_BOX * C::ROW);
            for (uint32_t i = 0; i < boxes; ++i)
                tma::tensor_g2s_2d(ring + slot * C::STAGE + i * AXC_BOX * C::ROW, &v_map, (int)(kvh * hd + d0), (int)(tile * AXC_T + i * AXC_BOX), full + slot);
        }
        // no copy may be in flight into this CTA's memory once it is gone, also when something gave up (the slot's other arrival may then be
        // missing: the limit, some milliseconds, is what the copy itself has)
        for (uint32_t t = tile > C::STAGES ? tile - C::STAGES : 0; t < tile; ++t)
            for (uint32_t i = 0; i < (1u << 16) && !tma::mbar_test(full + t % C::STAGES, (t / C::STAGES) & 1); ++i) __nanosleep(40);
        return;
    }
    if (warp >= AXC_HEADS) {
        // 1 / sum of the CTA's heads: lane-strided partials of the sums per AX_EPOS positions, then xor shuffles
        float inv[AXC_HEADS];
#pragma unroll
        for (int hh = 0; hh < AXC_HEADS; ++hh) {
            const float *parts = aux + (size_t)(kvh * G + h0 + min((uint32_t)hh, nh - 1)) * ld + ax_sums_at(ld);
            double tot = 0.0;
            for (uint32_t i = lane; i < (seq + AX_EPOS - 1) / AX_EPOS; i += 32)
                tot += __hiloint2double(__float_as_int(parts[2 * i]), __float_as_int(parts[2 * i + 1]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
            inv[hh] = (float)(1.0 / tot);
        }
        for (uint32_t tile = warp - AXC_HEADS; tile < n_tiles; tile += AXC_PWARPS) {
            const uint32_t slot = tile % C::STAGES, t0 = tile * AXC_T, cnt = min((uint32_t)AXC_T, seq - t0);
            float e[AXC_HEADS][AXC_T / 32];
#pragma unroll
            for (uint32_t hh = 0; hh < AXC_HEADS; ++hh)
#pragma unroll
                for (uint32_t i = 0; i < AXC_T / 32; ++i)
                    e[hh][i] = hh < nh && 32 * i + lane < cnt ? ws[(size_t)(kvh * G + h0 + hh) * ld + t0 + 32 * i + lane] : 0.0f;
            if (tile >= C::STAGES && !tma::mbar_wait_warp(empty + slot, (tile / C::STAGES - 1) & 1, &gave_up, &g_ax_status, 2u)) return;
            char *dst = ring + slot * C::STAGE;
            float *pd = reinterpret_cast<float *>(dst + C::V_BYTES);
#pragma unroll
            for (uint32_t hh = 0; hh < AXC_HEADS; ++hh)  // p = e * (1 / sum), rounded, as the reference stores it
#pragma unroll
                for (uint32_t i = 0; i < AXC_T / 32; ++i) pd[hh * AXC_T + 32 * i + lane] = __fmul_rn(e[hh][i], inv[hh]);
            const size_t row_bytes = (size_t)n_kv * hd * (F16 ? 2 : 4);
            const char *src = reinterpret_cast<const char *>(vc) + ((size_t)kvh * hd + d0) * (F16 ? 2 : 4) + (size_t)t0 * row_bytes;
            constexpr uint32_t PIECES = C::ROW / 16;
            for (uint32_t i = cnt / AXC_BOX * AXC_BOX * PIECES + lane; i < cnt * PIECES; i += 32) ax_cp16(dst + (size_t)i * 16, src + i / PIECES * row_bytes + i % PIECES * 16);
            ax_commit();
            ax_wait<0>();
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(full + slot);
        }
        return;
    }
    if (warp >= nh) return;
    float acc = 0.0f;
    for (uint32_t tile = 0; tile < n_tiles; ++tile) {
        const uint32_t slot = tile % C::STAGES;
        if (!tma::mbar_wait_warp(full + slot, (tile / C::STAGES) & 1, &gave_up, &g_ax_status, 1u)) return;
        const uint32_t base = tma::smem_u32(ring + slot * C::STAGE);
        acc = ax_chain<F16>(base, base + C::V_BYTES + warp * AXC_T * 4, min((uint32_t)AXC_T, seq - tile * AXC_T), acc);
        __syncwarp();
        if (lane == 0) tma::mbar_arrive(empty + slot);
    }
    acc = ax_by_dim<F16>(acc, lane);
    ax_emit(acc, (size_t)(kvh * G + h0 + warp) * hd + d0 + lane, lane, out, scales, quants, sums, tp);
}

// ONE launch for contexts of up to 1024 positions: a thread-block cluster per KV head, (hd / 32) x HS CTAs; a CTA walks the chains of
// 32 dims of HC = ceil(G / HS) heads.  Every CTA computes the scores of its share of the positions for all heads and stores
// them into the tables of the CTAs that walk those heads (distributed shared memory); after one cluster barrier each CTA runs
// the softmax on its own table and then the chains.  All of V's slice is requested at the start (cp.async) and lands meanwhile;
// the share's K rows come the same way, in whole lines, padded by 16 bytes so that eight rows are read without bank conflicts.
// 32 heads of 128 in groups of 4, f32, 512 / 1024 positions: 9.5 / 12.9 us alone (12.4 / 18 with four heads per CTA, K rows read
// in 32-byte pieces and chains that waited for their loads).
// f32 heads of 256 in groups of 7 or 8 do not fit its shared memory and take three launches: 13.8 / 16.3 us at 300 / 1000 positions, 16 heads
// of 2 KV heads (with half the K rows staged they fit, 9.8 / 24.1 us).
// grid = n_kv * cluster size CTAs, AX_VTHREADS threads; dynamic shared memory: AxFused.
template <int HD, bool F16>
struct AxFused {
    static constexpr uint32_t ES = F16 ? 2 : 4, KROWS = 128 * 128 / HD, KSTRIDE = HD * ES + 16;  // K rows staged at a time
    static constexpr uint32_t K_BYTES = KROWS * KSTRIDE;
    static size_t smem(uint32_t pos, uint32_t G, uint32_t HC) { return (size_t)pos * 32 * ES + K_BYTES + ((size_t)(pos + 4) * HC + (size_t)G * HD) * 4; }
};
template <int HD, bool F16>
__global__ void __launch_bounds__(AX_VTHREADS, 1)
attn_fused_exact_kernel(const float *__restrict__ q, const void *__restrict__ kc, const void *__restrict__ vc, int vec, uint32_t seq_len,
                        const uint32_t *__restrict__ seq_dev, uint32_t n_kv, uint32_t G, uint32_t HC, float scale, uint32_t smem_pos,
                        float *__restrict__ out, float *scales, int8_t *quants, int16_t *sums, const TpHook tp) {
    using F = AxFused<HD, F16>;
    extern __shared__ __align__(16) char axf_dyn[];
    constexpr uint32_t SL = HD / 32, WARPS = AX_VTHREADS / 32, ES = F::ES;  // SL: slices of a head
    char *vt = axf_dyn;                                  // [smem_pos][32]
    char *kt = vt + (size_t)smem_pos * 32 * ES;          // [KROWS][KSTRIDE]
    float *ax_p = reinterpret_cast<float *>(kt + F::K_BYTES);  // [HC][smem_pos + 4]
    const uint32_t pstride = smem_pos + 4;
    float *ax_q = ax_p + (size_t)HC * pstride;           // [G][HD]
    __shared__ double red_d[WARPS];
    __shared__ float red_f[WARPS];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t CL = cluster.num_blocks(), r = cluster.block_rank(), kvh = blockIdx.x / CL, d0 = r % SL * 32, h0 = r / SL * HC, nh = min(HC, G - h0);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a CTA's shared memory may be written by its peers only once it runs: every CTA arrives here, and waits for the
    // others just before its first remote store
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    pdl_trigger();
    pdl_wait();
    uint32_t seq = seq_dev ? *seq_dev : seq_len;
    if (seq > smem_pos) seq = smem_pos;  // the score tables hold smem_pos positions; the host plans launches for the lengths they meet
    const size_t row_bytes = (size_t)n_kv * HD * ES;
    const uint32_t share = (seq + CL - 1) / CL, t_begin = min(seq, r * share), t_end = min(seq, t_begin + share);
    auto stage_k = [&](uint32_t t0) {
        const uint32_t rows = min(F::KROWS, t_end - t0);
        const char *src = reinterpret_cast<const char *>(kc) + (size_t)t0 * row_bytes + (size_t)kvh * HD * ES;
        constexpr uint32_t PIECES = HD * ES / 16;
        if (vec) {
            for (uint32_t i = tid; i < rows * PIECES; i += AX_VTHREADS) ax_cp16(kt + i / PIECES * F::KSTRIDE + i % PIECES * 16, src + i / PIECES * row_bytes + i % PIECES * 16);
        } else {  // a cache that does not start on a 16-byte boundary
            for (uint32_t i = tid; i < rows * HD; i += AX_VTHREADS) {
                char *d = kt + i / HD * F::KSTRIDE + i % HD * ES;
                const char *g = src + i / HD * row_bytes + i % HD * ES;
                if (F16) *reinterpret_cast<uint16_t *>(d) = __ldg(reinterpret_cast<const uint16_t *>(g));
                else *reinterpret_cast<uint32_t *>(d) = __ldg(reinterpret_cast<const uint32_t *>(g));
            }
        }
        ax_commit();
    };
    if (t_begin < t_end) stage_k(t_begin);
    else ax_commit();
    {
        const char *src = reinterpret_cast<const char *>(vc) + ((size_t)kvh * HD + d0) * ES;
        constexpr uint32_t PIECES = 32 * ES / 16;
        for (uint32_t i = tid; i < seq * PIECES; i += AX_VTHREADS) ax_cp16(vt + (size_t)i * 16, src + i / PIECES * row_bytes + i % PIECES * 16);
        ax_commit();
    }
    for (uint32_t i = tid; i < G * HD; i += AX_VTHREADS) ax_q[i] = q[(size_t)kvh * G * HD + i];
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // ---- scores of this CTA's share of the positions: sixteen positions per warp, lanes p and p + 16 take position p
    for (uint32_t tk = t_begin; tk < t_end; tk += F::KROWS) {
        if (tk > t_begin) {
            __syncthreads();  // everyone is done with the rows staged before
            stage_k(tk);
            ax_wait<0>();
        } else {
            ax_wait<1>();
        }
        __syncthreads();
        const uint32_t a = lane >> 4, rows = min(F::KROWS, t_end - tk), tiles = (rows + 15) / 16;
        // where the tiles leave warps idle, the heads are dealt out too
        const uint32_t hs = min(max(WARPS / tiles, 1u), G);
        for (uint32_t item = warp; item < tiles * hs; item += WARPS) {
            const uint32_t row = item / hs * 16 + (lane & 15);
            const char *kr = kt + min(row, rows - 1) * F::KSTRIDE + 8 * a * ES;
            float k[HD / 16][8];
            auto load = [&] {
#pragma unroll
                for (int j = 0; j < HD / 16; ++j) {
                    if constexpr (F16) {
                        const uint4 w = *reinterpret_cast<const uint4 *>(kr + 32 * j);
                        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int i = 0; i < 8; ++i) k[j][i] = h2f((uint16_t)(ww[i / 2] >> (16 * (i & 1))));
                    } else {
                        const float4 lo = *reinterpret_cast<const float4 *>(kr + 64 * j), hi = *reinterpret_cast<const float4 *>(kr + 64 * j + 16);
                        k[j][0] = lo.x, k[j][1] = lo.y, k[j][2] = lo.z, k[j][3] = lo.w;
                        k[j][4] = hi.x, k[j][5] = hi.y, k[j][6] = hi.z, k[j][7] = hi.w;
                    }
                }
            };
            if (HD <= 128) load();
#pragma unroll 1
            for (uint32_t h = item % hs; h < G; h += hs) {
                if (HD > 128) load();  // 128 values do not stay in registers
                const float sc = ax_score<HD, 16>(ax_q + h * HD, k, a, scale);
                const uint32_t first = h / HC * SL;  // the CTAs of this head
#pragma unroll
                for (uint32_t c = 0; c < SL; c += 2)
                    if (row < rows && c + a < SL) cluster.map_shared_rank(ax_p, first + c + a)[(size_t)(h % HC) * pstride + tk + row] = sc;
            }
        }
    }
    cluster.sync();  // every CTA's table is complete; nothing remote is touched after this point

    // ---- probabilities of the CTA's heads.  Head h is handled by warps [h * nwh, (h + 1) * nwh).
    const uint32_t nwh = WARPS / HC, h_mine = warp / nwh, wl = warp % nwh;  // warps past nh * nwh idle here
    const bool has_head = h_mine < nh;
    const uint32_t hth = nwh * 32, hti = wl * 32 + lane;  // threads of my head, my index among them
    float *p_row = ax_p + (size_t)(has_head ? h_mine : 0) * pstride;
    float mx = -INFINITY;
    if (has_head) {
#pragma unroll 4
        for (uint32_t t = hti; t < seq; t += hth) mx = fmaxf(mx, p_row[t]);  // f32::max fold: NaN scores are ignored
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red_f[warp] = mx;
    __syncthreads();
    if (has_head) {
        mx = red_f[h_mine * nwh];
        for (uint32_t w = 1; w < nwh; ++w) mx = fmaxf(mx, red_f[h_mine * nwh + w]);
    }
    // exponentials and their f64 sum (fixed tree: thread-strided partials, xor shuffles, the head's warps in index order)
    double sum = 0.0;
    if (has_head) {
#pragma unroll 4
        for (uint32_t t = hti; t < seq; t += hth) {
            const float e = ggml_expf(__fsub_rn(p_row[t], mx));
            p_row[t] = e;
            sum += (double)e;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) red_d[warp] = sum;
    __syncthreads();
    if (has_head) {
        double tot = red_d[h_mine * nwh];
        for (uint32_t w = 1; w < nwh; ++w) tot += red_d[h_mine * nwh + w];
        const float inv = (float)(1.0 / tot);
#pragma unroll 4
        for (uint32_t t = hti; t < seq; t += hth) p_row[t] = __fmul_rn(p_row[t], inv);
    }
    ax_wait<0>();  // this thread's part of V has landed
    __syncthreads();

    // ---- out[d] = fma(p[t], V[t][d], out[d]) in position order: warp h walks head h, a lane per output dim
    if (warp >= nh) return;
    const float acc = ax_by_dim<F16>(ax_chain<F16>(tma::smem_u32(vt), tma::smem_u32(ax_p + (size_t)warp * pstride), seq, 0.0f), lane);
    ax_emit(acc, (size_t)(kvh * G + h0 + warp) * HD + d0 + lane, lane, out, scales, quants, sums, tp);
}

constexpr size_t AX_SMEM_MAX = 226 * 1024;  // dynamic shared memory the values / fused kernels may ask for

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int HD, bool F16>
int32_t launch_fused(size_t smem, cudaStream_t st, const float *q, const void *kc, const void *vc, uint32_t seq_len, const uint32_t *seq_dev,
                     uint32_t nkv, uint32_t G, uint32_t HC, float scale, uint32_t fpos, float *out, float *scales, int8_t *quants, int16_t *sums,
                     const TpHook &tp) {
    const uint32_t cl = HD / 32 * ((G + HC - 1) / HC);
    static thread_local int raised_dev = -1;  // per instantiation: opt in to more than 48 KB once per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (raised_dev != dev) {
        CERA_CUDA_TRY(cudaFuncSetAttribute(attn_fused_exact_kernel<HD, F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AX_SMEM_MAX));
        raised_dev = dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nkv * cl);
    cfg.blockDim = dim3(AX_VTHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch();
    return check_cuda(cudaLaunchKernelEx(&cfg, attn_fused_exact_kernel<HD, F16>, q, kc, vc, (int)aligned16(kc), seq_len, seq_dev, nkv, G, HC, scale, fpos, out,
                                         scales, quants, sums, tp),
                      "attention (fused) launch");
}

template <int HD, bool F16>
int32_t launch_scores(dim3 grid, cudaStream_t st, const float *q, const void *kc, uint32_t seq_len, const uint32_t *seq_dev, uint32_t nkv, uint32_t G,
                      float scale, float *ws, float *aux, uint32_t ld) {
    return check_cuda(launch_k(attn_scores_exact_kernel<HD, F16>, grid, dim3(AX_SWARPS * 32), (size_t)G * HD * sizeof(float), st, q, kc, (int)aligned16(kc),
                               seq_len, seq_dev, nkv, G, scale, ws, aux, ld),
                      "attention (scores) launch");
}

template <bool F16>
int32_t launch_scores_hd(uint32_t hd, dim3 grid, cudaStream_t st, const float *q, const void *kc, uint32_t seq_len, const uint32_t *seq_dev, uint32_t nkv,
                         uint32_t G, float scale, float *ws, float *aux, uint32_t ld) {
    switch (hd) {
        case 32: return launch_scores<32, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 64: return launch_scores<64, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 96: return launch_scores<96, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 128: return launch_scores<128, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 160: return launch_scores<160, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 192: return launch_scores<192, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 224: return launch_scores<224, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        case 256: return launch_scores<256, F16>(grid, st, q, kc, seq_len, seq_dev, nkv, G, scale, ws, aux, ld);
        default: return fail(CERA_CUDA_ERR_UNSUPPORTED, "decode_attention: head_dim %u", hd);
    }
}

template <bool F16>
int32_t launch_chain(cudaStream_t st, const float *ws, const float *aux, uint32_t ld, uint32_t reach, const void *vc, uint32_t seq_len,
                     const uint32_t *seq_dev, uint32_t nkv, uint32_t G, uint32_t hd, float *out, float *scales, int8_t *quants, int16_t *sums, const TpHook &tp) {
    constexpr size_t smem = AxChain<F16>::SMEM;
    static thread_local int raised_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (raised_dev != dev) {
        CERA_CUDA_TRY(cudaFuncSetAttribute(attn_chain_exact_kernel<F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        raised_dev = dev;
    }
    CUtensorMap v_map;
    CERA_TRY(tensor_map_2d(&v_map, F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, F16 ? 2 : 4, vc, reach, (uint64_t)nkv * hd, 32,
                           AXC_BOX, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE));
    return check_cuda(launch_k(attn_chain_exact_kernel<F16>, dim3(hd / 32, nkv, (G + AXC_HEADS - 1) / AXC_HEADS), dim3(AXC_THREADS), smem, st,
                               v_map, ws, aux, ld, vc, seq_len, seq_dev, nkv, G, hd, out, scales, quants, sums, tp),
                      "attention (values) launch");
}

// CERA_CUDA_ATTN=flash (or any of the split-kernel selectors) keeps decode attention on the online-softmax kernels.
bool exact_off() {
    static const bool v = [] {
        const char *e = getenv("CERA_CUDA_ATTN");
        return e && e[0] != 0;
    }();
    return v;
}

}  // namespace

bool attn_exact_supports(size_t n_heads, size_t n_kv_heads, size_t head_dim) {
    if (exact_off() || n_kv_heads == 0 || n_heads % n_kv_heads) return false;
    const size_t G = n_heads / n_kv_heads;
    return G >= 1 && G <= 8 && head_dim % 32 == 0 && head_dim >= 32 && head_dim <= 256;
}

// Plan word of the reference-order kernels: ATT_EXACT_FLAG | b, b = 1..4: launches that serve up to b * 1024 positions (b = 1: in
// one launch); b = 5: as many as the workspace holds.
constexpr uint32_t ATT_EXACT_FLAG = 0x200;

uint32_t attn_exact_plan(size_t seq_len_hint) {
    const size_t b = (seq_len_hint + 1023) / 1024;
    return ATT_EXACT_FLAG | (uint32_t)(b < 1 ? 1 : b > 4 ? 5 : b);
}

size_t attn_exact_workspace_bytes(size_t n_heads, size_t seq_len) {
    return 2 * n_heads * ((seq_len + 63) / 64 * 64) * sizeof(float);
}

// The workspace's capacity fixes the row stride of the score matrix, so launches captured once (length read from
// seq_len_dev) serve every length the workspace can hold.
int32_t launch_decode_attention_exact(const float *q, const void *kc, const void *vc, int kv_f16, size_t n_heads, size_t n_kv_heads,
                                      size_t head_dim, size_t seq_len, const uint32_t *seq_len_dev, uint32_t plan, float scale,
                                      float *out, void *workspace, size_t workspace_bytes, float *scales, int8_t *quants,
                                      int16_t *sums, cudaStream_t st, const TpHook *tp) {
    if (!q || !kc || !vc || !out || !workspace) return fail(CERA_CUDA_ERR_BAD_ARG, "decode_attention: null argument");
    if (!aligned16(vc)) return fail(CERA_CUDA_ERR_BAD_ARG, "decode_attention: the value cache does not start on a 16-byte boundary");
    const size_t cap = workspace_bytes / (2 * n_heads * sizeof(float)) / 64 * 64;  // positions the workspace holds
    if (cap == 0 || seq_len > cap)
        return fail(CERA_CUDA_ERR_BAD_ARG, "decode_attention: workspace of %zu bytes holds %zu positions, %zu needed", workspace_bytes, cap, seq_len);
    if (seq_len == 0 && !seq_len_dev) return fail(CERA_CUDA_ERR_BAD_ARG, "decode_attention: empty KV cache");
    const uint32_t G = (uint32_t)(n_heads / n_kv_heads), hd = (uint32_t)head_dim, nkv = (uint32_t)n_kv_heads;
    const uint32_t ld = (uint32_t)cap;
    const uint32_t b = plan & 0xFF;
    size_t reach = b >= 5 ? cap : (size_t)b * 1024;  // longest length this launch may meet
    if (reach > cap) reach = cap;
    if (seq_len > reach) return fail(CERA_CUDA_ERR_BAD_ARG, "decode_attention: plan 0x%x does not cover %zu positions", plan, seq_len);
    float *ws = (float *)workspace, *aux = ws + n_heads * (size_t)ld;
    // ---- one launch when the scores fit shared memory (CERA_CUDA_ATTN_EXACT=split keeps the three-kernel form)
    static const bool no_fused = [] { const char *e = getenv("CERA_CUDA_ATTN_EXACT"); return e && strcmp(e, "split") == 0; }();
    if (!no_fused && b == 1 && (hd == 64 || hd == 128 || hd == 256)) {  // up to 1024 positions
        const uint32_t fpos = (uint32_t)reach, sl = (uint32_t)seq_len;
        const TpHook hook = tp ? *tp : TpHook{};
        uint32_t hs = 1;  // CTAs that share a slice's heads: two heads each if the cluster (at most 8) allows
        while (2 * hs * (hd / 32) <= 8 && 2 * hs <= (G + 1) / 2) hs *= 2;
        const uint32_t hc = (G + hs - 1) / hs;
#define CERA_AX_FUSED(HD, F16)                                                                                                        \
    if (hd == HD && (kv_f16 != 0) == F16 && AxFused<HD, F16>::smem(fpos, G, hc) <= AX_SMEM_MAX)                                          \
    return launch_fused<HD, F16>(AxFused<HD, F16>::smem(fpos, G, hc), st, q, kc, vc, sl, seq_len_dev, nkv, G, hc, scale, fpos, out, scales, \
                                 quants, sums, hook)
        CERA_AX_FUSED(64, true);
        CERA_AX_FUSED(64, false);
        CERA_AX_FUSED(128, true);
        CERA_AX_FUSED(128, false);
        CERA_AX_FUSED(256, true);
        CERA_AX_FUSED(256, false);
#undef CERA_AX_FUSED
    }
    // scores: a fixed number of CTAs per KV head walks the position tiles, so one captured launch serves every length
    const uint32_t tiles = (uint32_t)((reach + 16 * AX_SWARPS - 1) / (16 * AX_SWARPS)), sl = (uint32_t)seq_len;
    uint32_t per_head = (uint32_t)(2 * sm_count() / (int)nkv);
    if (per_head < 1) per_head = 1;
    if (per_head > tiles) per_head = tiles;
    const TpHook hook = tp ? *tp : TpHook{};
    count_launch(3);
    const dim3 sgrid(per_head, nkv);
    CERA_TRY(kv_f16 ? launch_scores_hd<true>(hd, sgrid, st, q, kc, sl, seq_len_dev, nkv, G, scale, ws, aux, ld)
                    : launch_scores_hd<false>(hd, sgrid, st, q, kc, sl, seq_len_dev, nkv, G, scale, ws, aux, ld));
    // exponentials: likewise, about four CTAs per SM
    uint32_t parts = (uint32_t)((reach + AX_EPOS - 1) / AX_EPOS);
    const uint32_t part_ctas = (uint32_t)(4 * sm_count() / (int)n_heads);
    if (parts > part_ctas) parts = part_ctas ? part_ctas : 1;
    CERA_TRY(check_cuda(launch_k(attn_exp_exact_kernel, dim3(parts, (unsigned)n_heads), dim3(AX_ETHREADS), 0, st, ws, aux,
                                 ld, sl, seq_len_dev),
                        "attention (exponentials) launch"));
    return kv_f16 ? launch_chain<true>(st, ws, aux, ld, (uint32_t)reach, vc, sl, seq_len_dev, nkv, G, hd, out, scales, quants, sums, hook)
                  : launch_chain<false>(st, ws, aux, ld, (uint32_t)reach, vc, sl, seq_len_dev, nkv, G, hd, out, scales, quants, sums, hook);
}

static const bool g_ax_status_registered = register_kernel_status([] {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_ax_status, sizeof(v));
    return (uint32_t)v << 23;  // bits 23, 24
});

}  // namespace cera

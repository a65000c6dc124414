// Causal attention of a chunk of prompt tokens (prefill), in f32 accuracy: on the tensor cores over an f16 cache, with FMAs over an
// f32 cache.
//
// f16: a CTA owns one KV head and 64 rows, a row = (query, head of the group), so every staged K / V row serves all of them.
// A warp holds its sixteen queries in registers and walks the keys in tiles of 64 as flash attention does: scores, running softmax,
// weighted values.  The products are mma.sync on f16: the cache's values as they are; a query and a probability enter as a high and a
// low f16, 22 bits, so that a product is two MMAs, the low one first, and its sums are truncated at full size by the second half
// only.  Queries are scaled by a power of two per row, probabilities by 2^14; what f16 then cannot tell from zero is 2^-39 of the row's
// largest |q| and of 1.  A tile's weighted values start from zero and are added to the running output in f32.
// What bounds it: the latency of a warp's own MMAs and exponentials, 256 and 32 a lane per 16 rows x 64 keys, with two warps per scheduler - 255
// registers - to hide it (tensor pipe 37 % active at 2047 tokens).  It stays on mma.sync because scores, probabilities and their halves
// live in registers between the two products.
// 32 heads of 128 in groups of 4: 512 tokens 50 us (153 with FMAs on the CUDA cores), 2047 tokens 345 us (1125).  Error against 64
// bits 3.0e-7 (4.0e-7).
//
// f32: a split into f16 halves would need scales, and one value far from the others' size - a key that the query does not even
// see, where a tile shares the scale - would cost the rest their bits.  These products stay in f32 (attn_prefill_tiled_kernel).
//
// Infinities and NaN: a row that ends without finite values - a probability of zero times an infinite value of a key it does not
// see, or an infinity split into halves - is computed again by attend_row, which reads no key past the row's limit.
//
// Arithmetic contract: cera/src/backend/cpu.rs:4028-4241 (scaled dot, causal limit start_pos + j, online softmax);
// the f32 summation order is this kernel's own.
#include <cuda_fp16.h>

#include <cstdlib>
#include <cstring>

#include "act.cuh"
#include "attention_row.cuh"
#include "mma.cuh"
#include "ops.h"

namespace cera {

namespace {

template <int HD>
struct Pa {
    static constexpr int TK = 64;           // keys per tile
    static constexpr int ROW = HD * 2 + 16; // bytes of a staged row: eight rows of an ldmatrix hit all banks
    static constexpr int TILE = TK * ROW;
    static constexpr size_t SMEM = 2 * 2 * TILE;  // [stage][K, V]
};

// Nothing infinite, no NaN?
template <int N>
__device__ __forceinline__ bool pa_finite(const float (&v)[N], float l) {
    float z = l * 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) z = fmaf(v[i], 0.0f, z);
    return z == 0.0f;
}

// The warp's rows whose bit is set in `again` once more.
template <int VEC, bool F16>
__device__ __forceinline__ void pa_again(uint32_t again, uint32_t r_first, uint32_t G, const float *q, const uint8_t *kc, const uint8_t *vc, uint32_t n_heads,
                                      uint32_t n_kv_heads, uint32_t start_pos, float scale, float *out) {
    for (; again; again &= again - 1) {
        const uint32_t r = r_first + __ffs(again) - 1;
        attend_row<VEC, F16>(q, kc, vc, n_heads, n_kv_heads, r / G, blockIdx.x * G + r % G, start_pos, scale, out);
    }
}

// Biased exponent of the power of two that brings values up to mx (its float's bits) below 2^14; 254 - it is the inverse's.
__device__ __forceinline__ uint32_t pa_up(uint32_t mx_bits) {
    const uint32_t e = mx_bits >> 23;
    return min(267u - e, 253u);
}
__device__ __forceinline__ float pa_pow2(uint32_t biased) { return __uint_as_float(biased << 23); }

template <int HD, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) attn_prefill_mma_kernel(const float *__restrict__ q, const uint8_t *__restrict__ kc,
                                                                      const uint8_t *__restrict__ vc, uint32_t n_heads, uint32_t n_kv_heads, uint32_t n,
                                                                      uint32_t start_pos, float scale, float *__restrict__ out) {
    using S = Pa<HD>;
    extern __shared__ __align__(16) uint8_t pa_smem[];
    constexpr int TK = S::TK, NT = TK / 8, KS = HD / 16, KK = TK / 16, ND = HD / 8, THREADS = WARPS * 32;
    constexpr int PIECES = HD * 2 / 16;  // 16-byte pieces of a cache row
    pdl_trigger();
    pdl_wait();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kvh = blockIdx.x, G = n_heads / n_kv_heads;
    const uint32_t rows = n * G, r_cta = (gridDim.y - 1 - blockIdx.y) * WARPS * 16;  // the longest rows start first
    const size_t kv_dim = (size_t)n_kv_heads * HD, q_dim = (size_t)n_heads * HD;
    const uint32_t cta_kv = start_pos + (min(r_cta + WARPS * 16, rows) - 1) / G + 1;  // keys the CTA's last query sees
    const uint32_t n_tiles = (cta_kv + TK - 1) / TK;
    const uint8_t *k_src = kc + (size_t)kvh * HD * 2, *v_src = vc + (size_t)kvh * HD * 2;

    auto issue = [&](uint32_t t) {
        uint8_t *kd = pa_smem + (t & 1) * 2 * S::TILE, *vd = kd + S::TILE;
        for (uint32_t i = tid; i < TK * PIECES; i += THREADS) {
            const uint32_t r = i / PIECES, pc = i % PIECES;
            const size_t src = (size_t)min(t * TK + r, cta_kv - 1) * kv_dim * 2 + pc * 16;  // rows past the limit are masked; keep the read in range
            tma::cp_async16(kd + r * S::ROW + pc * 16, k_src + src);
            tma::cp_async16(vd + r * S::ROW + pc * 16, v_src + src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);

    // ---- queries of the warp's rows, as A fragments: rows g and g + 8, columns 16 ks + 2 c + {0, 1, 8, 9}
    const uint32_t g = lane >> 2, c = lane & 3, r_warp = r_cta + warp * 16;
    const bool live = r_warp < rows;
    uint32_t qh[KS][4], ql[KS][4];
    float qf[2];      // 2^-u of both rows
    uint32_t lim[2];  // last key of both rows
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t r = min(r_warp + g + 8 * h, rows - 1);
        lim[h] = start_pos + r / G;
        const float *src = q + (size_t)(r / G) * q_dim + ((size_t)kvh * G + r % G) * HD + 2 * c;
        float2 v[KS][2];
        float mx = 0.0f;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                v[ks][j] = *reinterpret_cast<const float2 *>(src + 16 * ks + 8 * j);
                mx = fmaxf(mx, fmaxf(fabsf(v[ks][j].x), fabsf(v[ks][j].y)));
            }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const uint32_t up = pa_up(__float_as_uint(mx));
        const float f = pa_pow2(up);
        qf[h] = pa_pow2(254u - up);
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int j = 0; j < 2; ++j) split_f16(v[ks][j].x * f, v[ks][j].y * f, qh[ks][2 * j + h], ql[ks][2 * j + h]);
    }

    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f}, o[ND][4];
#pragma unroll
    for (int i = 0; i < ND; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = 0.0f;
    const uint32_t warp_kv = live ? start_pos + (min(r_warp + 16, rows) - 1) / G + 1 : 0;

    for (uint32_t t = 0; t < n_tiles; ++t) {
        if (t + 1 < n_tiles) {
            issue(t + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint8_t *kt = pa_smem + (t & 1) * 2 * S::TILE, *vt = kt + S::TILE;
        if (t * TK < warp_kv) {
            // ---- scores: keys 8 nt + 2 c + {0, 1} of rows g (0, 1) and g + 8 (2, 3)
            float s[NT][4];
            const uint8_t *kl = kt + (lane & 7) * S::ROW + (lane >> 3) * 16;
            // two key groups side by side, so that an MMA does not wait for the one before it
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2) {
                float u[2][4];  // the second half of the high products on its own: fewer truncations, more chains
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[nt + p][j] = u[p][j] = 0.0f;
                uint32_t b[2][KS / 2][4];
#pragma unroll
                for (int k2 = 0; k2 < KS / 2; ++k2)
#pragma unroll
                    for (int p = 0; p < 2; ++p) ldsm4(b[p][k2], kl + (nt + p) * 8 * S::ROW + k2 * 64);
#pragma unroll
                for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                    for (int p = 0; p < 2; ++p) mma_f16(s[nt + p], ql[ks], b[p][ks / 2][2 * (ks & 1)], b[p][ks / 2][2 * (ks & 1) + 1]);
#pragma unroll
                for (int ks = 0; ks < KS / 2; ++ks)
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        constexpr int H = KS / 2;
                        mma_f16(s[nt + p], qh[ks], b[p][ks / 2][2 * (ks & 1)], b[p][ks / 2][2 * (ks & 1) + 1]);
                        mma_f16(u[p], qh[H + ks], b[p][(H + ks) / 2][2 * (ks & 1)], b[p][(H + ks) / 2][2 * (ks & 1) + 1]);
                    }
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[nt + p][j] += u[p][j];
            }
            // ---- running softmax
            const uint32_t key0 = t * TK + 2 * c;
            float mx[2] = {-INFINITY, -INFINITY}, corr[2];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool seen = key0 + 8 * nt + (j & 1) <= lim[j >> 1];
                    s[nt][j] = seen ? __fmul_rn(s[nt][j] * qf[j >> 1], scale) : -INFINITY;
                    mx[j >> 1] = fmaxf(mx[j >> 1], s[nt][j]);
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
                mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
                const float m_new = fmaxf(m_run[h], mx[h]);  // finite: key 0 is seen by every row
                corr[h] = m_run[h] == -INFINITY ? 0.0f : ggml_expf(__fsub_rn(m_run[h], m_new));
                m_run[h] = m_new;
                l_run[h] *= corr[h];
            }
            uint32_t ph[KK][4], pl[KK][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float p[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const bool seen = key0 + 8 * nt + j <= lim[h];
                        p[j] = seen ? ggml_expf(__fsub_rn(s[nt][2 * h + j], m_run[h])) : 0.0f;
                        l_run[h] += p[j];
                    }
                    split_f16(p[0] * 16384.0f, p[1] * 16384.0f, ph[nt / 2][2 * (nt & 1) + h], pl[nt / 2][2 * (nt & 1) + h]);
                }
            // ---- weighted values: dims 8 nd + 2 c + {0, 1}
            const uint8_t *vl = vt + ((lane >> 3) * 8 + (lane & 7)) * S::ROW;
            constexpr int W = 4;  // groups of dims side by side
#pragma unroll
            for (int nd = 0; nd < ND; nd += W) {
                float a[W][4];
#pragma unroll
                for (int p = 0; p < W; ++p)
#pragma unroll
                    for (int j = 0; j < 4; ++j) a[p][j] = 0.0f;
                uint32_t b[W][KK / 2][4];
#pragma unroll
                for (int k2 = 0; k2 < KK / 2; ++k2)
#pragma unroll
                    for (int p = 0; p < W; ++p) ldsm4_trans(b[p][k2], vl + k2 * 32 * S::ROW + (nd + p) * 16);
#pragma unroll
                for (int kk = 0; kk < KK; ++kk)
#pragma unroll
                    for (int p = 0; p < W; ++p) mma_f16(a[p], pl[kk], b[p][kk / 2][2 * (kk & 1)], b[p][kk / 2][2 * (kk & 1) + 1]);
#pragma unroll
                for (int kk = 0; kk < KK; ++kk)
#pragma unroll
                    for (int p = 0; p < W; ++p) mma_f16(a[p], ph[kk], b[p][kk / 2][2 * (kk & 1)], b[p][kk / 2][2 * (kk & 1) + 1]);
#pragma unroll
                for (int p = 0; p < W; ++p)
#pragma unroll
                    for (int j = 0; j < 4; ++j) o[nd + p][j] = fmaf(a[p][j], 1.0f / 16384.0f, o[nd + p][j] * corr[j >> 1]);
            }
        }
        __syncthreads();  // the stage is refilled by the copy issued in the next iteration
    }

    uint32_t again = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
        const uint32_t r = r_warp + g + 8 * h;
        float v[2 * ND];
#pragma unroll
        for (int nd = 0; nd < ND; ++nd) v[2 * nd] = o[nd][2 * h], v[2 * nd + 1] = o[nd][2 * h + 1];
        uint32_t bad = r < rows && !pa_finite(v, l_run[h]) ? 1u << (g + 8 * h) : 0;
        again |= __reduce_or_sync(0xffffffffu, bad);
        if (r >= rows) continue;
        const float inv = 1.0f / l_run[h];
        float *dst = out + (size_t)(r / G) * q_dim + ((size_t)kvh * G + r % G) * HD + 2 * c;
#pragma unroll
        for (int nd = 0; nd < ND; ++nd) *reinterpret_cast<float2 *>(dst + 8 * nd) = make_float2(v[2 * nd] * inv, v[2 * nd + 1] * inv);
    }
    __syncwarp();  // a row's first values are not stored after its second
    if (again) pa_again<HD / 32, true>(again, r_warp, G, q, kc, vc, n_heads, n_kv_heads, start_pos, scale, out);
}

template <int HD>
int32_t launch_mma(const float *q, const uint8_t *kc, const uint8_t *vc, uint32_t nh, uint32_t nkv, uint32_t n, uint32_t sp, float scale, float *out,
                   cudaStream_t st) {
    constexpr size_t smem = Pa<HD>::SMEM;
    constexpr int WARPS = 4;  // 64 rows per CTA, two CTAs on an SM
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        CERA_CUDA_TRY(cudaFuncSetAttribute(attn_prefill_mma_kernel<HD, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured_dev = dev;
    }
    const dim3 grid(nkv, (unsigned)(((size_t)n * (nh / nkv) + WARPS * 16 - 1) / (WARPS * 16)));
    count_launch();
    return check_cuda(launch_k(attn_prefill_mma_kernel<HD, WARPS>, grid, dim3(WARPS * 32), smem, st, q, kc, vc, nh, nkv, n, sp, scale, out),
                      "prefill attention (tensor cores) launch");
}

// ---- f32 cache ----------------------------------------------------------------------------------------------------------
// A CTA owns one KV head and PA_BQ consecutive queries; warp w owns query w with all G heads of the group.  Keys go by in tiles of
// 32, double-buffered with cp.async:
//   scores : lane = key.  The lane keeps 32 dims of its K row in registers at a time and reads the queries as
//            shared-memory broadcasts: no shuffle per key, four FMAs per broadcast load.
//   softmax: one running maximum / sum per (query, head), updated once per tile (two warp reductions and ONE expf per
//            key, against a reduction and two expf per key in the one-warp-per-row kernel).
//   P.V    : lane = four output dims.  The tile's probabilities sit in shared memory, V rows are read as float4 and
//            shared by the G heads.
// Rows are padded to 132 floats, so the lane = key reads (stride one row) hit all 32 banks.
// 32 heads of 128 in groups of 4: 512 tokens 100 us, 2047 tokens 1366 us.  Error against 64 bits 5.7e-7.
constexpr int PA_WARPS = 8, PA_THREADS = PA_WARPS * 32, PA_BQ = PA_WARPS;
constexpr int PA_TK = 32;        // keys per tile
constexpr int PA_HD = 128;       // head dim
constexpr int PA_ROW = 528;      // bytes per staged row (512 of data + padding)

template <int G>
constexpr size_t pa_smem_bytes() {
    return (size_t)2 * 2 * PA_TK * PA_ROW + (size_t)(PA_BQ * G * PA_HD + PA_WARPS * G * PA_TK) * sizeof(float);
}

__device__ __forceinline__ float pa_warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <int G>
__global__ void __launch_bounds__(PA_THREADS) attn_prefill_tiled_kernel(const float *__restrict__ q, const uint8_t *__restrict__ kc,
                                                                        const uint8_t *__restrict__ vc, uint32_t n_heads,
                                                                        uint32_t n_kv_heads, uint32_t n, uint32_t start_pos,
                                                                        float scale, float *__restrict__ out) {
    extern __shared__ __align__(16) uint8_t pa_smem[];
    constexpr int ROWB = PA_ROW, ESZ = 4, STAGE = PA_TK * ROWB;
    constexpr int PIECES = PA_HD * ESZ / 16;          // 16-byte pieces per cache row
    uint8_t *ks = pa_smem;                            // [2][32][ROWB]
    uint8_t *vs = ks + 2 * STAGE;                     // [2][32][ROWB]
    float *qs = reinterpret_cast<float *>(vs + 2 * STAGE);   // [PA_BQ * G][128]
    float *ps = qs + PA_BQ * G * PA_HD;               // [warps][G][32]

    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t kvh = blockIdx.x;
    const uint32_t qb = gridDim.y - 1 - blockIdx.y;   // the longest rows start first
    const uint32_t q0 = qb * PA_BQ, j = q0 + warp;
    const size_t kv_dim = (size_t)n_kv_heads * PA_HD, q_dim = (size_t)n_heads * PA_HD;
    const uint32_t q_last = min(q0 + PA_BQ, n) - 1;
    const uint32_t cta_kv = start_pos + q_last + 1;   // keys the block's last query sees
    const uint32_t n_tiles = (cta_kv + PA_TK - 1) / PA_TK;
    const bool live = j < n;
    const uint32_t my_kv = live ? start_pos + j + 1 : 0;

    auto issue = [&](uint32_t t, int stage) {
        uint8_t *kd = ks + stage * STAGE, *vd = vs + stage * STAGE;
        for (int i = tid; i < PA_TK * PIECES; i += PA_THREADS) {
            const int r = i / PIECES, pc = i % PIECES;
            const uint32_t key = min(t * PA_TK + r, cta_kv - 1);   // rows past the limit are masked; keep the read in range
            const size_t src = ((size_t)key * kv_dim + (size_t)kvh * PA_HD) * ESZ + pc * 16;
            tma::cp_async16(kd + r * ROWB + pc * 16, kc + src);
            tma::cp_async16(vd + r * ROWB + pc * 16, vc + src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    issue(0, 0);
    // queries of the block: pair (w, g) at qs[(w * G + g) * 128]
    for (int i = tid; i < PA_BQ * G * 32; i += PA_THREADS) {
        const int pair = i >> 5, pc = i & 31;
        const uint32_t jq = q0 + pair / G;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (jq < n) v = *reinterpret_cast<const float4 *>(q + jq * q_dim + ((size_t)kvh * G + pair % G) * PA_HD + pc * 4);
        *reinterpret_cast<float4 *>(qs + pair * PA_HD + pc * 4) = v;
    }

    float m_run[G], l_run[G];
    float4 acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m_run[g] = -INFINITY;
        l_run[g] = 0.0f;
        acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float *qw = qs + warp * G * PA_HD;
    float *pw = ps + warp * G * PA_TK;

    for (uint32_t t = 0; t < n_tiles; ++t) {
        const int stage = t & 1;
        if (t + 1 < n_tiles) {
            issue(t + 1, stage ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (t * PA_TK < my_kv) {
            const uint8_t *kt = ks + stage * STAGE + lane * ROWB;
            const uint8_t *vt = vs + stage * STAGE;
            float2 s[G];
#pragma unroll
            for (int g = 0; g < G; ++g) s[g] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int dc = 0; dc < PA_HD / 32; ++dc) {
                float4 kr[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) kr[i] = *reinterpret_cast<const float4 *>(kt + (dc * 32 + 4 * i) * 4);
#pragma unroll
                for (int g = 0; g < G; ++g) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 qq = *reinterpret_cast<const float4 *>(qw + g * PA_HD + dc * 32 + 4 * i);
                        // packed f32 pairs (FFMA2): even dims accumulate in .x, odd dims in .y
                        s[g] = __ffma2_rn(make_float2(qq.x, qq.y), make_float2(kr[i].x, kr[i].y), s[g]);
                        s[g] = __ffma2_rn(make_float2(qq.z, qq.w), make_float2(kr[i].z, kr[i].w), s[g]);
                    }
                }
            }
            const bool valid = t * PA_TK + lane < my_kv;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float sv = valid ? __fmul_rn(__fadd_rn(s[g].x, s[g].y), scale) : -INFINITY;
                const float m_new = fmaxf(m_run[g], pa_warp_max(sv));   // finite: key t * 32 is valid for this query
                const float corr = m_run[g] == -INFINITY ? 0.0f : ggml_expf(__fsub_rn(m_run[g], m_new));
                const float p = valid ? ggml_expf(__fsub_rn(sv, m_new)) : 0.0f;
                l_run[g] = fmaf(l_run[g], corr, warp_sum(p));
                acc[g].x *= corr;
                acc[g].y *= corr;
                acc[g].z *= corr;
                acc[g].w *= corr;
                m_run[g] = m_new;
                pw[g * PA_TK + lane] = p;
            }
            __syncwarp();
#pragma unroll
            for (int k4 = 0; k4 < PA_TK / 4; ++k4) {
                const float4 v0 = *reinterpret_cast<const float4 *>(vt + (4 * k4 + 0) * ROWB + 16 * lane);
                const float4 v1 = *reinterpret_cast<const float4 *>(vt + (4 * k4 + 1) * ROWB + 16 * lane);
                const float4 v2 = *reinterpret_cast<const float4 *>(vt + (4 * k4 + 2) * ROWB + 16 * lane);
                const float4 v3 = *reinterpret_cast<const float4 *>(vt + (4 * k4 + 3) * ROWB + 16 * lane);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float4 pp = *reinterpret_cast<const float4 *>(pw + g * PA_TK + 4 * k4);
                    const float2 p0 = make_float2(pp.x, pp.x), p1 = make_float2(pp.y, pp.y), p2 = make_float2(pp.z, pp.z),
                                 p3 = make_float2(pp.w, pp.w);
                    float2 lo = make_float2(acc[g].x, acc[g].y), hi = make_float2(acc[g].z, acc[g].w);
                    lo = __ffma2_rn(p3, make_float2(v3.x, v3.y), __ffma2_rn(p2, make_float2(v2.x, v2.y),
                         __ffma2_rn(p1, make_float2(v1.x, v1.y), __ffma2_rn(p0, make_float2(v0.x, v0.y), lo))));
                    hi = __ffma2_rn(p3, make_float2(v3.z, v3.w), __ffma2_rn(p2, make_float2(v2.z, v2.w),
                         __ffma2_rn(p1, make_float2(v1.z, v1.w), __ffma2_rn(p0, make_float2(v0.z, v0.w), hi))));
                    acc[g] = make_float4(lo.x, lo.y, hi.x, hi.y);
                }
            }
            __syncwarp();   // the probabilities are rewritten by the next tile
        }
        __syncthreads();    // the stage is refilled by the copy issued in the next iteration
    }

    if (!live) return;
    uint32_t again = 0;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const float v[4] = {acc[g].x, acc[g].y, acc[g].z, acc[g].w}, inv = 1.0f / l_run[g];
        if (__any_sync(0xffffffffu, !pa_finite(v, l_run[g]))) again |= 1u << g;
        *reinterpret_cast<float4 *>(out + j * q_dim + ((size_t)kvh * G + g) * PA_HD + 4 * lane) = make_float4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
    }
    if (again) pa_again<PA_HD / 32, false>(again, j * G, G, q, kc, vc, n_heads, n_kv_heads, start_pos, scale, out);
}

template <int G>
int32_t launch_tiled(const float *q, const uint8_t *kc, const uint8_t *vc, uint32_t nh, uint32_t nkv, uint32_t n, uint32_t sp,
                     float scale, float *out, cudaStream_t st) {
    constexpr size_t smem = pa_smem_bytes<G>();
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        CERA_CUDA_TRY(cudaFuncSetAttribute(attn_prefill_tiled_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured_dev = dev;
    }
    const dim3 grid(nkv, (n + PA_BQ - 1) / PA_BQ);
    count_launch();
    return check_cuda(launch_k(attn_prefill_tiled_kernel<G>, grid, dim3(PA_THREADS), smem, st, q, kc, vc, nh, nkv, n, sp, scale, out),
                      "prefill attention (tiled) launch");
}

}  // namespace

// f16 cache: head_dim 64 or 128, any group size; f32 cache: head_dim 128, group size 1, 2, 4 or 8.  16-byte aligned operands; anything
// else: *taken = false and the caller runs the one-warp-per-row kernel.  CERA_CUDA_PREFILL_ATTN=rows turns these kernels off.
int32_t launch_prefill_attention_tiled(const float *q, const void *kc, const void *vc, int kv_f16, size_t n_heads,
                                       size_t n_kv_heads, size_t head_dim, size_t n, size_t start_pos, float scale, float *out,
                                       cudaStream_t st, bool *taken) {
    *taken = false;
    static const bool off = [] {
        const char *e = getenv("CERA_CUDA_PREFILL_ATTN");
        return e && strcmp(e, "rows") == 0;
    }();
    if (off || n == 0) return CERA_CUDA_OK;
    if (((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc | (uintptr_t)out) % 16) return CERA_CUDA_OK;
    const uint32_t nh = (uint32_t)n_heads, nkv = (uint32_t)n_kv_heads, nn = (uint32_t)n, sp = (uint32_t)start_pos;
    const uint8_t *kf = (const uint8_t *)kc, *vf = (const uint8_t *)vc;
    *taken = true;
    if (kv_f16 && head_dim == 128) return launch_mma<128>(q, kf, vf, nh, nkv, nn, sp, scale, out, st);
    if (kv_f16 && head_dim == 64) return launch_mma<64>(q, kf, vf, nh, nkv, nn, sp, scale, out, st);
    if (!kv_f16 && head_dim == PA_HD) switch (n_heads / n_kv_heads) {
            case 1: return launch_tiled<1>(q, kf, vf, nh, nkv, nn, sp, scale, out, st);
            case 2: return launch_tiled<2>(q, kf, vf, nh, nkv, nn, sp, scale, out, st);
            case 4: return launch_tiled<4>(q, kf, vf, nh, nkv, nn, sp, scale, out, st);
            case 8: return launch_tiled<8>(q, kf, vf, nh, nkv, nn, sp, scale, out, st);
        }
    *taken = false;
    return CERA_CUDA_OK;
}

}  // namespace cera

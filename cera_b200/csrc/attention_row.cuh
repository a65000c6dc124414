// Causal attention of one (query head, query token) by one warp in f32: the general path of prompts, and what the tiled kernels
// (attention_prefill.cu) fall back on for a row that met an infinity or a NaN.
#pragma once

#include <cuda_fp16.h>

#include "act.cuh"

namespace cera {

template <int VEC, bool F16>
__device__ __forceinline__ void load_row(const void *base, size_t elem_off, float (&v)[VEC]) {
    if (F16) {
        const __half *p = reinterpret_cast<const __half *>(base) + elem_off;
        if (VEC == 4) {
            const uint2 u = *reinterpret_cast<const uint2 *>(p);
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
            const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
            v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
        } else {
#pragma unroll
            for (int i = 0; i < VEC; i += 2) {
                const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(p + i));
                v[i] = a.x;
                v[i + 1] = a.y;
            }
        }
    } else {
        const float *p = reinterpret_cast<const float *>(base) + elem_off;
        if (VEC % 4 == 0) {
#pragma unroll
            for (int i = 0; i < VEC; i += 4) {
                const float4 a = *reinterpret_cast<const float4 *>(p + i);
                v[i] = a.x; v[i + 1] = a.y; v[i + 2] = a.z; v[i + 3] = a.w;
            }
        } else {
            const float2 a = *reinterpret_cast<const float2 *>(p);
            v[0] = a.x;
            v[1] = a.y;
        }
    }
}

// Online softmax over cache rows [0, start_pos + j] with the polynomial expf (cera/src/backend/cpu.rs:4146-4241; the tile
// width there is 32, here 1, which only changes f32 rounding).  Nothing past the limit is read.  q / out are token-major.
template <int VEC, bool F16>
__device__ __forceinline__ void attend_row(const float *__restrict__ q, const void *__restrict__ kc, const void *__restrict__ vc, uint32_t n_heads,
                                           uint32_t n_kv_heads, uint32_t j, uint32_t h, uint32_t start_pos, float scale, float *__restrict__ out) {
    constexpr int HD = VEC * 32;
    const int lane = threadIdx.x & 31;
    const uint32_t kvh = h / (n_heads / n_kv_heads);
    const size_t kv_dim = (size_t)n_kv_heads * HD, q_dim = (size_t)n_heads * HD;
    const size_t head_off = (size_t)kvh * HD + lane * VEC;
    float qv[VEC], acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
        qv[v] = q[j * q_dim + (size_t)h * HD + lane * VEC + v];
        acc[v] = 0.0f;
    }
    float m_run = -INFINITY, l_run = 0.0f;
    const uint32_t max_kv = start_pos + j + 1;
    for (uint32_t t0 = 0; t0 < max_kv; t0 += 4) {
        float kr[4][VEC], vr[4][VEC], sc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (t0 + i < max_kv) {
                load_row<VEC, F16>(kc, (t0 + i) * kv_dim + head_off, kr[i]);
                load_row<VEC, F16>(vc, (t0 + i) * kv_dim + head_off, vr[i]);
            } else {
#pragma unroll
                for (int v = 0; v < VEC; ++v) kr[i][v] = vr[i][v] = 0.0f;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float s = 0.0f;
#pragma unroll
            for (int v = 0; v < VEC; ++v) s = fmaf(qv[v], kr[i][v], s);
            sc[i] = s;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], o);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (t0 + i >= max_kv) break;
            const float s = __fmul_rn(sc[i], scale);
            const float m_new = fmaxf(m_run, s);
            const float corr = m_run == -INFINITY ? 0.0f : ggml_expf(__fsub_rn(m_run, m_new));
            const float pexp = ggml_expf(__fsub_rn(s, m_new));
            l_run = fmaf(l_run, corr, pexp);
#pragma unroll
            for (int v = 0; v < VEC; ++v) acc[v] = fmaf(pexp, vr[i][v], acc[v] * corr);
            m_run = m_new;
        }
    }
    const float inv = 1.0f / l_run;
#pragma unroll
    for (int v = 0; v < VEC; ++v) out[j * q_dim + (size_t)h * HD + lane * VEC + v] = acc[v] * inv;
}

}  // namespace cera

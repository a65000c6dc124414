// Device-side Q8_0 activation quantizer and the glue math it is fused with.
#pragma once

#include "common.cuh"

namespace cera {

// Q8_0-quantized activations as the kernels consume them (column j at j*k).
struct ActView {
    const float *scales;    // [n][k/32]
    const int8_t *quants;   // [n][k]
    const int16_t *sums;    // [n][k/16] sums of 16 consecutive quants
};

// ggml's polynomial expf, operation for operation (cera/src/backend/cpu.rs:2504-2544);
// every step individually rounded so the result is bit-identical to the CPU's.
__device__ __forceinline__ float ggml_expf(float x) {
    const float R = __uint_as_float(0x4B400000u), LOG2E = __uint_as_float(0x3FB8AA3Bu),
                LN2_HI = __uint_as_float(0x3F317200u), LN2_LO = __uint_as_float(0x35BFBE8Eu),
                C1 = __uint_as_float(0x3F7FFFF6u), C2 = __uint_as_float(0x3EFFFEDBu),
                C3 = __uint_as_float(0x3E2AAF33u), C4 = __uint_as_float(0x3D2B9F17u),
                C5 = __uint_as_float(0x3C072010u);
    const float z = __fadd_rn(R, __fmul_rn(x, LOG2E));
    const float n = __fsub_rn(z, R);
    const float b = __fsub_rn(__fsub_rn(x, __fmul_rn(n, LN2_HI)), __fmul_rn(n, LN2_LO));
    const uint32_t e = __float_as_uint(z) << 23;
    const float k = __uint_as_float(e + 0x3F800000u);
    const float u = __fmul_rn(b, b);
    const float p45 = __fadd_rn(C4, __fmul_rn(C5, b));
    const float p23 = __fadd_rn(__fadd_rn(C2, __fmul_rn(C3, b)), __fmul_rn(p45, u));
    const float j = __fadd_rn(__fmul_rn(C1, b), __fmul_rn(p23, u));
    const float abs_n = fabsf(n);
    if (abs_n <= 126.0f) return __fadd_rn(k, __fmul_rn(j, k));
    if (abs_n > 192.0f) return n > 0.0f ? __int_as_float(0x7F800000) : 0.0f;
    const uint32_t d = n <= 0.0f ? 0x82000000u : 0u;
    const float s1 = __uint_as_float(d + 0x7F000000u);
    const float s2 = __uint_as_float(e - d);
    return __fmul_rn(__fadd_rn(s2, __fmul_rn(s2, j)), s1);
}

// Two of them by packed instructions, which round each half as the plain ones do; outside of the polynomial's plain range one at a time.
__device__ __forceinline__ float2 ggml_expf2(float2 x) {
    auto c = [](uint32_t v) { return make_float2(__uint_as_float(v), __uint_as_float(v)); };
    const float2 z = __fadd2_rn(c(0x4B400000u), __fmul2_rn(x, c(0x3FB8AA3Bu)));
    const float2 n = __fadd2_rn(z, c(0xCB400000u));
    const float2 b = __fadd2_rn(__fadd2_rn(x, __fmul2_rn(n, c(0xBF317200u))), __fmul2_rn(n, c(0xB5BFBE8Eu)));
    const float2 k = make_float2(__uint_as_float((__float_as_uint(z.x) << 23) + 0x3F800000u), __uint_as_float((__float_as_uint(z.y) << 23) + 0x3F800000u));
    const float2 u = __fmul2_rn(b, b);
    const float2 p45 = __fadd2_rn(c(0x3D2B9F17u), __fmul2_rn(c(0x3C072010u), b));
    const float2 p23 = __fadd2_rn(__fadd2_rn(c(0x3EFFFEDBu), __fmul2_rn(c(0x3E2AAF33u), b)), __fmul2_rn(p45, u));
    const float2 j = __fadd2_rn(__fmul2_rn(c(0x3F7FFFF6u), b), __fmul2_rn(p23, u));
    float2 r = __fadd2_rn(k, __fmul2_rn(j, k));
    if (!(fabsf(n.x) <= 126.0f)) r.x = ggml_expf(x.x);
    if (!(fabsf(n.y) <= 126.0f)) r.y = ggml_expf(x.y);
    return r;
}

// cera/src/backend/cpu.rs:2573: g / (1 + expf(-g)) * u
__device__ __forceinline__ float silu_mul(float g, float u) {
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, ggml_expf(-g))), u);
}

__device__ __forceinline__ float2 silu_mul2(float2 g, float2 u) {
    const float2 d = __fadd2_rn(make_float2(1.0f, 1.0f), ggml_expf2(make_float2(-g.x, -g.y)));
    return __fmul2_rn(make_float2(__fdiv_rn(g.x, d.x), __fdiv_rn(g.y, d.y)), u);
}

// One warp quantizes one 32-element block: lane t holds v (cera/src/backend/cpu.rs:942-958).
// Returns the int8 quant of this lane; lane 0 of each 16-lane half gets the half sum in
// `half_sum`; `scale` is the f16-rounded block scale (same on every lane).
__device__ __forceinline__ int quantize_lane(float v, float &scale, int &half_sum) {
    float amax = fabsf(v);
    if (amax != amax) amax = 0.0f;  // f32::max ignores NaN
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float d = __fdiv_rn(amax, 127.0f);
    const float r = __fdiv_rn(1.0f, d);
    const float id = (d != 0.0f && isfinite(r)) ? r : 0.0f;
    scale = __half2float(__float2half_rn(d));
    float p = rintf(__fmul_rn(v, id));
    int q;
    if (p != p) q = 0;
    else q = (int)fminf(fmaxf(p, -128.0f), 127.0f);
    int s = q;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    half_sum = s;
    return q;
}

// The same block with four consecutive elements per lane: eight neighbouring lanes hold it, all of them in the call.
struct QuantQuad {
    uint32_t quants;  // four int8, the first lowest
    float scale;      // same on the eight lanes
    int half_sum;     // sum of the 16-element half this lane is in
};
__device__ __forceinline__ QuantQuad quantize_quad(const float (&e)[4]) {
    float amax = fmaxf(fmaxf(fabsf(e[0]), fabsf(e[1])), fmaxf(fabsf(e[2]), fabsf(e[3])));  // fmaxf, like f32::max, ignores NaN
    amax = amax == amax ? amax : 0.0f;                                                     // (four of them)
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float d = __fdiv_rn(amax, 127.0f);
    const float r = __fdiv_rn(1.0f, d);
    const float id = (d != 0.0f && isfinite(r)) ? r : 0.0f;
    // |e * id| is at most 127 and a few roundings, or NaN: added to 1.5 * 2^23 it is rounded to the nearest integer, ties to even, in the
    // low bits - without the conversions' slow pipe and with nothing to clamp
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float p = __fadd_rn(__fmul_rn(e[i], id), 12582912.0f);
        q[i] = p == p ? __float_as_uint(p) : 0x4B400000u;
    }
    const uint32_t quants = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
    int s4 = __dp4a((int)quants, 0x01010101, 0);
    s4 += __shfl_xor_sync(0xffffffffu, s4, 1);
    s4 += __shfl_xor_sync(0xffffffffu, s4, 2);
    return {quants, __half2float(__float2half_rn(d)), s4};
}

// The same for eight consecutive values a lane: a block is four neighbouring lanes, half the shuffles and divisions a value.
struct QuantOct {
    uint2 quants;
    float scale;   // same on the four lanes
    int half_sum;  // sum of the 16-element half this lane is in
};
__device__ __forceinline__ QuantOct quantize_oct(const float (&e)[8]) {
    float amax = 0.0f;  // fmaxf, like f32::max, ignores NaN
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(e[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d = __fdiv_rn(amax, 127.0f);
    const float r = __fdiv_rn(1.0f, d);
    const float id = (d != 0.0f && isfinite(r)) ? r : 0.0f;
    uint32_t q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // as in quantize_quad
        const float p = __fadd_rn(__fmul_rn(e[i], id), 12582912.0f);
        q[i] = p == p ? __float_as_uint(p) : 0x4B400000u;
    }
    QuantOct o;
    o.quants.x = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
    o.quants.y = __byte_perm(__byte_perm(q[4], q[5], 0x0040), __byte_perm(q[6], q[7], 0x0040), 0x5410);
    int s8 = __dp4a((int)o.quants.y, 0x01010101, __dp4a((int)o.quants.x, 0x01010101, 0));
    o.half_sum = s8 + __shfl_xor_sync(0xffffffffu, s8, 1);
    o.scale = __half2float(__float2half_rn(d));
    return o;
}

}  // namespace cera

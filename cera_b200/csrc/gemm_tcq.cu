// Batched product of quantized weights with Q8_0 columns on the fifth-generation tensor cores, straight from the quantized
// bytes: out[m x n] = W x X for Q4_0, Q4_1, Q8_0, and Q6_K, and for these, Q4_K and
// Q5_K the expert-grouped form of the routed feed-forward, two matrices (gate, up) at a time.
//
// The arithmetic of the formats scales the integer sum of every 32-element block by (weight scale) x (activation scale).  Both
// operands are integers that f16 holds exactly - the activation quants, and the weight quants, for K-quants times their
// six-bit (Q6_K: int8) sub-block scale - and so is every partial sum of a block in f32 (below 2^24), so two tcgen05.mma of
// K = 16 leave the block's exact sum in TMEM.  Q6_K's products have 13 bits: a rounded part and the remainder, two operands.
// The epilogue adds (d * xs) * sum to f32 registers, packed in pairs, and subtracts the minimum's term m * (xs * A), A the block's sum
// of quants.  Same operations and types as the kernels that form the sums with integer instructions, in the order of k: error against 64 bits
// 1.6e-7 to 2e-7 at k of 4096 to 14336 (mma.sync 2e-7; eight columns at a time, whose 32 lanes have shorter chains, 0.8e-7 to 1.1e-7).
//
// What bounds it: no unit's rate (tensor pipe 8 to 14 % active, issue slots 41 to 43 %, DRAM 10 %), but the hands a stage passes through: four warps convert its
// weights, and a thread per weight row makes each of their 16-byte loads touch 32 lines; then the products; then the rescale, two packed
// f32 instructions per pair of cells (three with a minimum) and 256 broadcasts of column scales.  4096 x 14336 Q6_K, 64 columns: 60 us
// (110 with mma.sync, which also spends the issue slots of its fragments); 14336 x 4096 Q8_0, 2048 columns: 1.08 ms (12.9 ms by eight
// columns at a time).
//
// A CTA is persistent: it walks units (128 rows x up to BN columns x a share of k), one warp issuing the products, one
// requesting activation tiles by bulk copies, four warps converting weights into the operand tiles, eight draining finished
// blocks.  A grid of units that would leave SMs idle splits k; the
// partial tiles go through a scratch buffer and are added in the order of k.  Every wait is bounded (tma.cuh).
//
// Arithmetic contract: cera/src/backend/simd.rs:5248-5371 (32-element blocks), 5693-5878 (Q4_K), 5988-6195 (Q6_K), per cell.
#include <cstdlib>
#include <cstring>

#include "act.cuh"
#include "gemv_task.cuh"
#include "ops.h"
#include "tc.cuh"
#include "tma.cuh"

namespace cera {

__device__ unsigned int g_tcq_status = 0;  // bits 0..3: products, activations, weights, epilogue gave up

namespace {

constexpr uint32_t TQ_BM = 128, TQ_KS = 64;  // rows of a tile, k of a stage: two blocks
constexpr uint32_t TQ_PROD = 4, TQ_EPI = 8, TQ_THREADS = (2 + TQ_EPI + TQ_PROD) * 32;
constexpr uint32_t TQ_IMG_THREADS = 512;  // 64 columns: a block each; with 256, two rounds, 4096 x 14336 Q6_K at 64 columns takes 69.5 us, 65.1 so
constexpr int TQ_SEGS = 2;
constexpr uint32_t TQ_COL = TQ_KS * 2 + 16;  // bytes a column takes in a stage: quants as f16, scale and scaled sum of both blocks

constexpr bool tq_kquant(int t) { return t == CERA_TYPE_Q4_K || t == CERA_TYPE_Q5_K || t == CERA_TYPE_Q6_K; }
constexpr bool tq_has_min(int t) { return t == CERA_TYPE_Q4_1 || t == CERA_TYPE_Q4_K || t == CERA_TYPE_Q5_K; }

template <int T, int BN>
struct Tq {
    static constexpr uint32_t KC = TQ_BM * 16, OP = 8 * KC, NA = T == CERA_TYPE_Q6_K ? 2 : 1;  // bytes between 8-element k chunks of a weight operand
    // a stage: weight operands, activation tile with the scales and scaled sums of both blocks, weight scales and minima of both
    static constexpr uint32_t X_BYTES = BN * TQ_COL, W_OFF = NA * OP + X_BYTES, STAGE = W_OFF + 4 * TQ_BM * 4;
    static constexpr uint32_t STAGES = 200 * 1024 / STAGE < 8 ? 200 * 1024 / STAGE : 8;
    static constexpr uint32_t TAIL = STAGES * STAGE, SMEM = TAIL + 256;
    static constexpr uint32_t ACC = BN == 128 ? 2 : 4, TMEM = ACC * 2 * BN;  // accumulators of a stage: two blocks of BN columns
};

struct TqParams {
    WeightView w[TQ_SEGS];  // matrices that take the same columns
    float *out[TQ_SEGS];
    uint32_t m[TQ_SEGS], ldc[TQ_SEGS];  // rows (grouped: of an expert); cell (i, j) at out[i * ldy + j * ldc]
    uint32_t tile_end[TQ_SEGS];         // row tiles up to and including the matrix
    uint32_t n, k, ldy;
    int epilogue;
    uint32_t row_tiles, col_tiles, splits, n_it, nb;  // of all matrices; of the columns; of k; 64s and 32s of k
    const uint8_t *img;    // activations: per (column tile, stage) quants as f16 [8 chunks][nc][8], then [block][scale, scale x sum of the quants][nc]
    float *partial;        // splits > 1: [split][row tile][column tile][BN][128]
    const MoeTile *tiles;  // grouped: column tile t is tiles[t]
    const uint32_t *n_tiles;
};

// One unit of work.
struct TqUnit {
    uint32_t seg, rt, all_rt, ct, split, s0, s1;  // matrix, row tile in it and among all, column tile, share of k: stages [s0, s1)
    uint32_t first, cnt, nc;                      // its columns; rounded up to a multiple of 16
    size_t w_row0;                                // first row in the weight
};
template <int BN>
__device__ __forceinline__ TqUnit tq_unit(const TqParams &p, uint32_t u) {
    TqUnit o;
    o.split = u % p.splits;
    u /= p.splits;
    uint32_t expert = 0;
    if (p.tiles) {  // all rows of a column tile side by side: its activation tiles stay in L2
        o.ct = u / p.row_tiles;
        o.rt = u % p.row_tiles;
        const MoeTile t = p.tiles[o.ct];
        expert = t.expert;
        o.first = t.first;
        o.cnt = t.count;
    } else {
        o.rt = u / p.col_tiles;
        o.ct = u % p.col_tiles;
        o.first = o.ct * BN;
        o.cnt = min((uint32_t)BN, p.n - o.first);
    }
    o.all_rt = o.rt;
    o.seg = o.rt < p.tile_end[0] ? 0 : 1;
    if (o.seg) o.rt -= p.tile_end[0];
    o.nc = (o.cnt + 15) & ~15u;
    const uint32_t pairs = (p.n_it + 1) / 2;  // k is split between 128s
    o.s0 = 2 * (uint32_t)((uint64_t)pairs * o.split / p.splits);
    o.s1 = min(p.n_it, 2 * (uint32_t)((uint64_t)pairs * (o.split + 1) / p.splits));
    o.w_row0 = (size_t)expert * p.m[o.seg] + o.rt * TQ_BM;
    return o;
}
__device__ __forceinline__ uint32_t tq_units(const TqParams &p) { return p.row_tiles * p.splits * (p.tiles ? *p.n_tiles : p.col_tiles); }

__device__ __forceinline__ void tq_bytes_to_h1024(uint32_t v, __half2 &lo, __half2 &hi) {  // 1024 + byte, four bytes
    const uint32_t a = __byte_perm(v, 0x64646464u, 0x5140), b = __byte_perm(v, 0x64646464u, 0x7362);
    lo = *reinterpret_cast<const __half2 *>(&a);
    hi = *reinterpret_cast<const __half2 *>(&b);
}

// ---- activations ------------------------------------------------------------------------------------------------------
// grid (column tiles, 256s of k): thread = (column, 32-element block).
template <int BN>
__global__ void __launch_bounds__(TQ_IMG_THREADS) tq_image_kernel(const ActView x, uint32_t n, uint32_t k, uint32_t n_it, const MoeTile *__restrict__ tiles,
                                                                   const uint32_t *__restrict__ n_tiles, uint8_t *__restrict__ img) {
    pdl_trigger();
    pdl_wait();
    const uint32_t ct = blockIdx.x, nb = k >> 5;
    uint32_t first = ct * BN, cnt;
    if (tiles) {
        if (ct >= *n_tiles) return;
        first = tiles[ct].first;
        cnt = tiles[ct].count;
    } else {
        cnt = min((uint32_t)BN, n - first);
    }
    const uint32_t nc = (cnt + 15) & ~15u;
    for (uint32_t i = threadIdx.x; i < nc * 8; i += TQ_IMG_THREADS) {
        const uint32_t c = i % nc, b = blockIdx.y * 8 + i / nc;
        if (b >= nb) break;
        uint4 r[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
        float sc = 0.0f;
        if (c < cnt) {
            const uint4 *src = reinterpret_cast<const uint4 *>(x.quants + (size_t)(first + c) * k + (size_t)b * 32);
            r[0] = __ldg(src);
            r[1] = __ldg(src + 1);
            sc = __ldg(x.scales + (size_t)(first + c) * nb + b);
        }
        const uint32_t words[8] = {r[0].x, r[0].y, r[0].z, r[0].w, r[1].x, r[1].y, r[1].z, r[1].w};
        int sum = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) sum = __dp4a((int)words[q], 0x01010101, sum);
        uint8_t *dst = img + ((size_t)ct * n_it * BN + (size_t)(b >> 1) * nc) * TQ_COL;
        float *dst_x = reinterpret_cast<float *>(dst + nc * (TQ_KS * 2)) + (b & 1) * 2 * nc + c;
        dst_x[0] = sc;
        dst_x[nc] = sc * (float)sum;
        dst += (b & 1) * 4 * nc * 16 + c * 16;
        const __half2 off = __float2half2_rn(-1152.0f);
#pragma unroll
        for (uint32_t ch = 0; ch < 4; ++ch) {
            __half2 h[4];
            tq_bytes_to_h1024(words[2 * ch] ^ 0x80808080u, h[0], h[1]);  // quant + 128
            tq_bytes_to_h1024(words[2 * ch + 1] ^ 0x80808080u, h[2], h[3]);
#pragma unroll
            for (int q = 0; q < 4; ++q) h[q] = __hadd2(h[q], off);
            *reinterpret_cast<uint4 *>(dst + ch * nc * 16) = *reinterpret_cast<const uint4 *>(&h[0]);
        }
    }
}

// ---- weights ----------------------------------------------------------------------------------------------------------
// What a producer thread (a row) reads for 128 elements of k, two stages, twice (half = 0, 1).
//   32-element formats: block 2 s + half of both stages s;  Q4_K / Q5_K: piece 2 s + half (low nibbles: 16 elements of the stage's
//   first block, high: of its second);  Q6_K: pieces half and 2 + half (stage s: their low or high nibbles).
template <int T>
struct TqRaw {
    uint4 q[T == CERA_TYPE_Q8_0 ? 4 : 2];
    uint4 qh;       // Q5_K, Q6_K: high bits
    uint4 h;        // K-quants: header (Q6_K: sixteen int8 scales)
    uint32_t d[2];  // 32-element formats: scale (and minimum) of both blocks; Q6_K: super-scale

    __device__ __forceinline__ void load(const WeightView &w, size_t row, uint32_t chunk, uint32_t half) {
        if constexpr (tq_kquant(T)) {
            const size_t sbi = sb_index(w, row, chunk >> 1);
            h = __ldg(reinterpret_cast<const uint4 *>(w.hdr) + sbi);
            if constexpr (T == CERA_TYPE_Q6_K) {
                q[0] = __ldg(reinterpret_cast<const uint4 *>(q_piece_ptr(w, row, 4, chunk * 4 + half)));
                q[1] = __ldg(reinterpret_cast<const uint4 *>(q_piece_ptr(w, row, 4, chunk * 4 + 2 + half)));
                qh = __ldg(reinterpret_cast<const uint4 *>(w.qh + sbi * 64 + (chunk & 1) * 32 + half * 16));
                d[0] = __ldg(reinterpret_cast<const uint16_t *>(w.d) + sbi);
            } else {
                q[0] = __ldg(reinterpret_cast<const uint4 *>(q_piece_ptr(w, row, 4, chunk * 4 + half)));
                q[1] = __ldg(reinterpret_cast<const uint4 *>(q_piece_ptr(w, row, 4, chunk * 4 + 2 + half)));
                if constexpr (T == CERA_TYPE_Q5_K) qh = __ldg(reinterpret_cast<const uint4 *>(w.qh + sbi * 32 + half * 16));
            }
        } else {
            constexpr uint32_t NP = T == CERA_TYPE_Q8_0 ? 8 : 4, PB = T == CERA_TYPE_Q8_0 ? 2 : 1;
#pragma unroll
            for (uint32_t s = 0; s < 2; ++s) {
                const uint32_t b = chunk * 4 + 2 * s + half;
                const bool in = b < w.nb;
#pragma unroll
                for (uint32_t i = 0; i < PB; ++i)
                    q[s * PB + i] = in ? __ldg(reinterpret_cast<const uint4 *>(q_piece_ptr(w, row, NP, b * PB + i))) : make_uint4(0, 0, 0, 0);
                if (T == CERA_TYPE_Q4_1) d[s] = in ? __ldg(reinterpret_cast<const uint32_t *>(w.hdr) + row * w.nb + b) : 0;
                else d[s] = in ? __ldg(reinterpret_cast<const uint16_t *>(w.hdr) + row * w.nb + b) : 0;
            }
        }
    }
};

// This thread's 32 weights of stage s (0, 1) of the chunk into the operand tile at `a` (Q6_K: remainders OP bytes behind), and the
// scale and minimum of one of the stage's blocks (block `half`) for the epilogue.
template <int T, int BN>
__device__ __forceinline__ void tq_convert(const TqRaw<T> &raw, uint32_t chunk, uint32_t s, uint32_t r, uint32_t half, uint8_t *a, float &scale, float &minimum) {
    using S = Tq<T, BN>;
    minimum = 0.0f;
    // eight integers (bytes, `off` too large) times a scale, as f16; REST: what the rounding left, exactly
    auto chunk8 = [&](uint32_t w0, uint32_t w1, __half2 o, __half2 sc, uint8_t *dst) {
        __half2 q[4];
        tq_bytes_to_h1024(w0, q[0], q[1]);
        tq_bytes_to_h1024(w1, q[2], q[3]);
        if constexpr (T == CERA_TYPE_Q6_K) {
            __half2 l[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __half2 v = __hadd2(q[i], o);
                q[i] = __hmul2_rn(v, sc);
                l[i] = __hfma2(v, sc, __hneg2(q[i]));
            }
            *reinterpret_cast<uint4 *>(dst + S::OP) = *reinterpret_cast<const uint4 *>(&l[0]);
        } else if constexpr (tq_kquant(T)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = __hfma2(q[i], sc, o);  // (1024 + q) sc - 1024 sc, an exact value rounded once
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = __hadd2(q[i], o);
        }
        *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(&q[0]);
    };
    if constexpr (T == CERA_TYPE_Q6_K) {
        // piece j holds elements 32 j + 16 half + [0, 16) of the stage
        const uint32_t hw[4] = {raw.qh.x, raw.qh.y, raw.qh.z, raw.qh.w}, scw[4] = {raw.h.x, raw.h.y, raw.h.z, raw.h.w};
        scale = h2f((uint16_t)raw.d[0]);
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            const uint32_t si = (chunk & 1) * 8 + (2 * s + j) * 2 + half;
            const uint32_t word = si < 8 ? (si < 4 ? scw[0] : scw[1]) : (si < 12 ? scw[2] : scw[3]);
            const __half2 sc = __half2half2(__int2half_rn((int)(int8_t)(word >> (8 * (si & 3)))));
            const uint32_t qw[4] = {raw.q[j].x, raw.q[j].y, raw.q[j].z, raw.q[j].w};
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = ((qw[i] >> (4 * s)) & 0x0F0F0F0Fu) | (((hw[i] >> (4 * s + 2 * j)) & 0x03030303u) << 4);
#pragma unroll
            for (uint32_t c = 0; c < 2; ++c) chunk8(v[2 * c], v[2 * c + 1], __float2half2_rn(-1056.0f), sc, a + (4 * j + 2 * half + c) * S::KC + r * 16);
        }
    } else if constexpr (tq_kquant(T)) {
        const uint32_t hf = chunk & 1;  // task of the super-block
        uint32_t scp, mnp;
        kq_quad(raw.h, hf, scp, mnp);
        scale = h2f((uint16_t)(raw.h.x & 0xFFFF));
        minimum = h2f((uint16_t)(raw.h.x >> 16)) * (float)((mnp >> (16 * s + 8 * half)) & 0xFF);
        const uint32_t qw[4] = {raw.q[s].x, raw.q[s].y, raw.q[s].z, raw.q[s].w}, hw[4] = {raw.qh.x, raw.qh.y, raw.qh.z, raw.qh.w};
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {  // low, high nibbles: the stage's first, second block
            const __half2 sc = __half2half2(__ushort2half_rn((unsigned short)((scp >> (16 * s + 8 * j)) & 0xFF)));
            const __half2 o = __hmul2(sc, __float2half2_rn(-1024.0f));
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[i] = (qw[i] >> (4 * j)) & 0x0F0F0F0Fu;
                if (T == CERA_TYPE_Q5_K) v[i] |= ((hw[i] >> (4 * hf + 2 * s + j)) & 0x01010101u) << 4;
            }
#pragma unroll
            for (uint32_t c = 0; c < 2; ++c) chunk8(v[2 * c], v[2 * c + 1], o, sc, a + (4 * j + 2 * half + c) * S::KC + r * 16);
        }
    } else {
        scale = h2f((uint16_t)(raw.d[s] & 0xFFFF));
        if (T == CERA_TYPE_Q4_1) minimum = -h2f((uint16_t)(raw.d[s] >> 16));
        uint8_t *dst = a + 4 * half * S::KC + r * 16;
        const __half2 o = __float2half2_rn(T == CERA_TYPE_Q8_0 ? -1152.0f : T == CERA_TYPE_Q4_0 ? -1032.0f : -1024.0f);
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) {
            if constexpr (T == CERA_TYPE_Q8_0) {
                const uint4 v = raw.q[2 * s + c / 2];
                chunk8((c & 1 ? v.z : v.x) ^ 0x80808080u, (c & 1 ? v.w : v.y) ^ 0x80808080u, o, o, dst + c * S::KC);
            } else {  // low nibbles: elements 0-15, high nibbles: 16-31
                const uint4 v = raw.q[s];
                chunk8(((c & 1 ? v.z : v.x) >> (c < 2 ? 0 : 4)) & 0x0F0F0F0Fu, ((c & 1 ? v.w : v.y) >> (c < 2 ? 0 : 4)) & 0x0F0F0F0Fu, o, o, dst + c * S::KC);
            }
        }
    }
}

template <int T, int BN>
__global__ void __launch_bounds__(TQ_THREADS, 1) gemm_tcq_kernel(const __grid_constant__ TqParams p) {
    using S = Tq<T, BN>;
    extern __shared__ __align__(1024) uint8_t tq_smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(tq_smem + S::TAIL);
    uint64_t *full = bars, *empty = bars + S::STAGES, *full_d = bars + 2 * S::STAGES, *empty_d = full_d + S::ACC;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(empty_d + S::ACC);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_trigger();
    if (tid == 0) {
        for (uint32_t s = 0; s < S::STAGES; ++s) {
            tma::mbar_init(full + s, 1 + TQ_PROD);  // the activation request's expect_tx, the producer warps
            tma::mbar_init(empty + s, 1 + TQ_EPI);  // the commit of the stage's products, the epilogue warps
        }
        for (uint32_t b = 0; b < S::ACC; ++b) {
            tma::mbar_init(full_d + b, 1);        // the commit
            tma::mbar_init(empty_d + b, TQ_EPI);  // every epilogue warp has read the accumulators
        }
        *abort_flag = 0;
        tma::mbar_init_fence();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, S::TMEM);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // only the weights, and without experts the units, are known before the kernels ahead have finished
    if (p.tiles || warp < 2 + TQ_EPI) pdl_wait();
    const uint32_t units = tq_units(p);
    uint32_t it = 0;  // stages so far, over all units

    if (warp == 0) {
        // ---- products: the whole warp, one lane issues
        const uint32_t me = elect_one();
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const TqUnit o = tq_unit<BN>(p, u);
            const uint32_t idesc = (1u << 4) | ((o.nc >> 3) << 17) | ((TQ_BM >> 4) << 24);  // f16 x f16 -> f32, K-major
            for (uint32_t st = o.s0; st < o.s1; ++st, ++it) {
                const uint32_t s = it % S::STAGES, b = it % S::ACC, nblk = min(2u, p.nb - 2 * st);
                ok = tma::mbar_wait_warp(empty_d + b, ((it / S::ACC) & 1) ^ 1, abort_flag, &g_tcq_status, 1u) &&
                     tma::mbar_wait_warp(full + s, (it / S::STAGES) & 1, abort_flag, &g_tcq_status, 1u);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a = tma::smem_u32(tq_smem + s * S::STAGE), x = a + S::NA * S::OP, d = tmem + b * 2 * BN;
                const uint64_t ad = smem_desc(a, S::KC, 128), xd = smem_desc(x, o.nc * 16, 128);  // address fields count 16 bytes
#pragma unroll
                for (uint32_t ks = 0; ks < 4; ++ks) {
                    const uint32_t on = ks / 2 < nblk ? me : 0;
                    tc_mma_f16(d + ks / 2 * BN, ad + 2 * ks * S::KC / 16, xd + 2 * ks * o.nc, idesc, ks & 1, on);
                    if (S::NA == 2) tc_mma_f16(d + ks / 2 * BN, ad + (S::OP + 2 * ks * S::KC) / 16, xd + 2 * ks * o.nc, idesc, 1, on);
                }
                tc_commit(full_d + b, me);
                tc_commit(empty + s, me);
            }
        }
    } else if (warp == 1) {
        // ---- activations: the whole warp, one lane requests
        const uint32_t me = elect_one();
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const TqUnit o = tq_unit<BN>(p, u);
            const uint8_t *src = p.img + (size_t)o.ct * p.n_it * BN * TQ_COL;
            const uint32_t bytes = o.nc * TQ_COL;
            for (uint32_t st = o.s0; st < o.s1; ++st, ++it) {
                const uint32_t s = it % S::STAGES;
                ok = tma::mbar_wait_warp(empty + s, ((it / S::STAGES) & 1) ^ 1, abort_flag, &g_tcq_status, 2u);
                if (!ok) break;
                tma::mbar_expect_tx_if(full + s, bytes, me);  // (of a last half stage no product and no sum reads the second block)
                tma::bulk_g2s_if(tq_smem + s * S::STAGE + S::NA * S::OP, src + (size_t)st * bytes, bytes, full + s, me);
            }
        }
        // this CTA's shared memory must outlive the copies in flight (they only are when something gave up)
        if (*abort_flag)
            for (uint32_t i = it > S::STAGES ? it - S::STAGES : 0; i < it; ++i)
                for (uint32_t n = 0; n < (1u << 16) && !tma::mbar_test(full + i % S::STAGES, (i / S::STAGES) & 1); ++n) __nanosleep(40);
    } else if (warp < 2 + TQ_EPI) {
        // ---- epilogue: lane = row, half of the columns, the running sums in registers
        const uint32_t quad = warp & 3, ch = (warp - 2) >> 2, c_base = ch * (BN / 2);
        const uint32_t rl = quad * 32 + lane, lane_addr = tmem + ((quad * 32) << 16);
        constexpr uint32_t CW = BN / 2 < 32 ? BN / 2 : 32;  // columns read at a time
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const TqUnit o = tq_unit<BN>(p, u);
            float2 acc[BN / 4];
#pragma unroll
            for (int i = 0; i < BN / 4; ++i) acc[i] = make_float2(0.0f, 0.0f);
            for (uint32_t st = o.s0; st < o.s1; ++st, ++it) {
                const uint32_t s = it % S::STAGES, b = it % S::ACC, nblk = min(2u, p.nb - 2 * st);
                ok = tma::mbar_wait_warp(full_d + b, (it / S::ACC) & 1, abort_flag, &g_tcq_status, 8u);
                if (!ok) break;
                tc_fence_after();
                const uint8_t *stage = tq_smem + s * S::STAGE;
                const float *wsc = reinterpret_cast<const float *>(stage + S::W_OFF) + rl;
                const float *xs = reinterpret_cast<const float *>(stage + S::NA * S::OP + o.nc * (TQ_KS * 2)) + c_base;
#pragma unroll
                for (uint32_t blk = 0; blk < 2; ++blk) {
                    if (blk >= nblk) break;
                    const float ds = wsc[blk * 2 * TQ_BM], mn = tq_has_min(T) ? -wsc[(blk * 2 + 1) * TQ_BM] : 0.0f;
                    const float2 ds2 = make_float2(ds, ds), mn2 = make_float2(mn, mn);
#pragma unroll
                    for (uint32_t c = 0; c < BN / 2; c += CW) {
                        if (c_base + c >= o.nc) break;
                        uint32_t v[CW / 16][16];
#pragma unroll
                        for (uint32_t i = 0; i < CW / 16; ++i) tmem_ld16(lane_addr + (b * 2 + blk) * BN + c_base + c + 16 * i, v[i]);  // (columns past nc: never added)
                        tmem_wait_ld();
                        const float4 *f4 = reinterpret_cast<const float4 *>(xs + blk * 2 * o.nc + c), *e4 = reinterpret_cast<const float4 *>(xs + (blk * 2 + 1) * o.nc + c);
#pragma unroll
                        for (int q = 0; q < (int)CW / 4; ++q) {
                            const float4 f = f4[q];
                            float2 &a0 = acc[c / 2 + 2 * q], &a1 = acc[c / 2 + 2 * q + 1];
                            if (tq_has_min(T)) {
                                const float4 e = e4[q];
                                a0 = __ffma2_rn(mn2, make_float2(e.x, e.y), a0);
                                a1 = __ffma2_rn(mn2, make_float2(e.z, e.w), a1);
                            }
                            a0 = __ffma2_rn(make_float2(__uint_as_float(v[q / 4][q % 4 * 4]), __uint_as_float(v[q / 4][q % 4 * 4 + 1])), __fmul2_rn(ds2, make_float2(f.x, f.y)), a0);
                            a1 = __ffma2_rn(make_float2(__uint_as_float(v[q / 4][q % 4 * 4 + 2]), __uint_as_float(v[q / 4][q % 4 * 4 + 3])), __fmul2_rn(ds2, make_float2(f.z, f.w)), a1);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    tma::mbar_arrive(empty_d + b);
                    tma::mbar_arrive(empty + s);
                }
            }
            if (!ok) break;
            const uint32_t row = o.rt * TQ_BM + rl;
            auto cell = [&](uint32_t c) { return c & 1 ? acc[c / 2].y : acc[c / 2].x; };
            if (p.splits > 1) {
                float *dst = p.partial + (((size_t)o.split * p.row_tiles + o.all_rt) * p.col_tiles + o.ct) * (BN * TQ_BM) + (size_t)c_base * TQ_BM + rl;
#pragma unroll
                for (uint32_t c = 0; c < BN / 2; ++c)
                    if (c_base + c < o.cnt) dst[(size_t)c * TQ_BM] = cell(c);
            } else if (row < p.m[o.seg]) {
                const uint32_t ldc = p.ldc[o.seg];
                float *dst = p.out[o.seg] + (size_t)row * p.ldy + (size_t)(o.first + c_base) * ldc;
                const bool vec = ldc == 1 && ((uintptr_t)dst & 15) == 0;
#pragma unroll
                for (uint32_t c = 0; c < BN / 2; c += 4) {
                    if (c_base + c >= o.cnt) break;
                    if (vec && p.epilogue != EPI_ADD && c_base + c + 4 <= o.cnt) {
                        *reinterpret_cast<float4 *>(dst + c) = make_float4(cell(c), cell(c + 1), cell(c + 2), cell(c + 3));
                        continue;
                    }
#pragma unroll
                    for (uint32_t i = c; i < c + 4; ++i)
                        if (c_base + i < o.cnt) {
                            float *d = dst + (size_t)i * ldc;
                            *d = p.epilogue == EPI_ADD ? __fadd_rn(*d, cell(i)) : cell(i);
                        }
                }
            }
        }
    } else {
        // ---- weights: thread = row, 128 elements of k fetched ahead of their conversion
        const uint32_t r = tid - (2 + TQ_EPI) * 32;
        struct Pos {
            uint32_t u, chunk, end, seg;  // unit; 128s of k
            size_t row;
        };
        auto enter = [&](Pos &o) {
            if (o.u >= units) return;
            const TqUnit t = tq_unit<BN>(p, o.u);
            o.chunk = t.s0 / 2;
            o.end = (t.s1 + 1) / 2;
            o.seg = t.seg;
            o.row = t.w_row0 + min(r, p.m[t.seg] - 1 - t.rt * TQ_BM);  // rows past the edge repeat the last one; their results are not stored
        };
        Pos cur{blockIdx.x, 0, 0, 0, 0};
        enter(cur);
        TqRaw<T> raw[2];
        auto load = [&](TqRaw<T>(&x)[2], const Pos &o) {
#pragma unroll
            for (uint32_t half = 0; half < 2; ++half) x[half].load(p.w[o.seg], o.row, o.chunk, half);
        };
        if (cur.u < units) load(raw, cur);
        bool ok = true;
        while (cur.u < units && ok) {
            Pos nx = cur;
            if (++nx.chunk >= nx.end) {
                nx.u += gridDim.x;
                enter(nx);
            }
            TqRaw<T> ahead[2];
            if (nx.u < units) load(ahead, nx);
#pragma unroll
            for (uint32_t st = 0; st < 2; ++st) {
                const uint32_t stage = 2 * cur.chunk + st;
                if (stage >= p.n_it) break;
                const uint32_t s = it % S::STAGES;
                ok = tma::mbar_wait_warp(empty + s, ((it / S::STAGES) & 1) ^ 1, abort_flag, &g_tcq_status, 4u);
                if (!ok) break;
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {
                    float sc, mn;
                    tq_convert<T, BN>(raw[half], cur.chunk, st, r, half, tq_smem + s * S::STAGE, sc, mn);
                    float *dst = reinterpret_cast<float *>(tq_smem + s * S::STAGE + S::W_OFF) + half * 2 * TQ_BM + r;
                    dst[0] = sc;
                    if (tq_has_min(T)) dst[TQ_BM] = mn;
                }
                fence_async_smem();  // the products read shared memory through the asynchronous proxy
                __syncwarp();
                if (lane == 0) tma::mbar_arrive(full + s);
                ++it;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) raw[h] = ahead[h];
            cur = nx;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, S::TMEM);
    }
}

// Adds the partial tiles in the order of k.  thread = (row, four columns).
template <int BN>
__global__ void __launch_bounds__(256) tq_reduce_kernel(const __grid_constant__ TqParams p) {
    pdl_trigger();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x, tile = i / (TQ_BM * BN / 4);
    const uint32_t r = i % TQ_BM, c = i / TQ_BM % (BN / 4) * 4;
    if (tile >= (size_t)p.row_tiles * p.col_tiles) return;
    uint32_t rt = (uint32_t)(tile / p.col_tiles);
    const uint32_t col = (uint32_t)(tile % p.col_tiles) * BN + c, seg = rt < p.tile_end[0] ? 0 : 1;
    if (seg) rt -= p.tile_end[0];
    const uint32_t row = rt * TQ_BM + r, ldc = p.ldc[seg];
    if (row >= p.m[seg] || col >= p.n) return;
    const float *src = p.partial + tile * (BN * TQ_BM) + (size_t)c * TQ_BM + r;
    const size_t step = (size_t)p.row_tiles * p.col_tiles * BN * TQ_BM;
    const uint32_t nc = min(4u, p.n - col);
    float v[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) v[j] = j < nc ? src[(size_t)j * TQ_BM] : 0.0f;
    for (uint32_t s = 1; s < p.splits; ++s)
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (j < nc) v[j] += src[s * step + (size_t)j * TQ_BM];
    float *o = p.out[seg] + (size_t)row * p.ldy + (size_t)col * ldc;
    if (ldc == 1 && nc == 4 && p.epilogue != EPI_ADD && ((uintptr_t)o & 15) == 0) {
        *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
        if (j < nc) o[(size_t)j * ldc] = p.epilogue == EPI_ADD ? __fadd_rn(o[(size_t)j * ldc], v[j]) : v[j];
}

// Splits of k for a product of so many 128-row x BN-column tiles, `pairs` 128s of k each: those expected to finish first, us: rounds of units on
// the SMs, each its share of k (measured per 128 of k: 2.15 with 128 columns, 1.7 with 64, 1.47 with 32), plus the reduction's launch and
// traffic.  Against every split from 1 to 16, at eight shapes from 1024 x 1024 x 64 to 4096 x 14336 x 512, the choice is within 1 % of the
// fastest, once within 4 % (4096 x 4096 x 128 Q8_0: 86 us whole, 35.3 in four as chosen, 49.7 in five).
uint32_t tcq_splits(uint64_t whole, uint32_t pairs, uint32_t bn) {
    const uint32_t sms = (uint32_t)sm_count();
    const double tp = 1.25 + 0.007 * bn, cells = (double)whole * bn * TQ_BM;
    double best = 1e30;
    uint32_t splits = 1;
    for (uint32_t s = 1; s <= 16 && 2 * s <= pairs + 1; ++s) {
        const double rounds = (double)((whole * s + sms - 1) / sms);
        const double t = rounds * (((pairs + s - 1) / s) * tp + 1.0) + (s > 1 ? 2.5 + cells * 4 * (s + 1) / 3e6 : 0.0);
        if (t < best) {
            best = t;
            splits = s;
        }
    }
    return splits;
}

// A plain product whose converted activations would take more than this goes through them in parts of the columns.
constexpr size_t TQ_IMG_LIMIT = 256ull << 20;

// The scratch of col_tiles column tiles: activations, then the partial tiles of a split.
template <int BN>
size_t tcq_bytes(const TqParams &p, uint32_t col_tiles, size_t *img_bytes, uint32_t *splits) {
    const uint64_t whole = (uint64_t)p.row_tiles * col_tiles;
    *splits = p.tiles ? 1 : tcq_splits(whole, (p.n_it + 1) / 2, BN);
    *img_bytes = (size_t)col_tiles * p.n_it * BN * TQ_COL;
    return *img_bytes + (*splits > 1 ? (size_t)*splits * whole * BN * TQ_BM * 4 : 0);
}

template <int T, int BN>
int32_t launch_tcq_part(TqParams p, const ActView &x, uint8_t *scratch, cudaStream_t st) {
    size_t img_bytes;
    tcq_bytes<BN>(p, p.col_tiles, &img_bytes, &p.splits);
    p.img = scratch;
    p.partial = reinterpret_cast<float *>(scratch + img_bytes);
    count_launch(2);
    CERA_TRY(check_cuda(launch_k(tq_image_kernel<BN>, dim3(p.col_tiles, (p.k + 255) / 256), dim3(TQ_IMG_THREADS), 0, st, x, p.n, p.k, p.n_it, p.tiles,
                                 p.n_tiles, scratch),
                        "gemm (quantized, tcgen05) activation launch"));
    const uint64_t whole = (uint64_t)p.row_tiles * p.col_tiles, units = whole * p.splits, sms = (uint64_t)sm_count();
    CERA_TRY(check_cuda(launch_k(gemm_tcq_kernel<T, BN>, dim3((unsigned)(units < sms ? units : sms)), dim3(TQ_THREADS), (size_t)Tq<T, BN>::SMEM, st, p),
                        "gemm (quantized, tcgen05) launch"));
    if (p.splits == 1) return CERA_CUDA_OK;
    count_launch();
    return check_cuda(launch_k(tq_reduce_kernel<BN>, dim3((unsigned)((whole * (BN / 4) * TQ_BM + 255) / 256)), dim3(256), 0, st, p),
                      "gemm (quantized, tcgen05) reduction launch");
}

template <int T, int BN>
int32_t launch_tcq_bn(TqParams p, int segs, const ActView &x, uint32_t max_col_tiles, uint8_t *given, cudaStream_t st, bool *taken) {
    p.row_tiles = 0;
    for (int i = 0; i < TQ_SEGS; ++i) {
        if (i < segs) p.row_tiles += (p.m[i] + TQ_BM - 1) / TQ_BM;
        p.tile_end[i] = p.row_tiles;
    }
    p.n_it = (p.k + TQ_KS - 1) / TQ_KS;
    p.nb = p.k / 32;
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        CERA_CUDA_TRY(cudaFuncSetAttribute(gemm_tcq_kernel<T, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Tq<T, BN>::SMEM));
        configured_dev = dev;
    }
    if (given) {
        *taken = true;
        p.col_tiles = max_col_tiles;
        return launch_tcq_part<T, BN>(p, x, given, st);
    }
    const size_t most = TQ_IMG_LIMIT / ((size_t)p.n_it * BN * TQ_COL);
    const uint32_t part = most < 1 ? 1 : most < max_col_tiles ? (uint32_t)most : max_col_tiles, last = (max_col_tiles - 1) % part + 1;
    size_t img;
    uint32_t splits;
    const size_t bytes = tcq_bytes<BN>(p, part, &img, &splits), bytes_last = tcq_bytes<BN>(p, last, &img, &splits);
    uint8_t *scratch = (uint8_t *)scratch_alloc(bytes > bytes_last ? bytes : bytes_last, st);
    if (!scratch) return CERA_CUDA_OK;  // no room for the operands: leave the product to the kernels that need none
    *taken = true;
    int32_t rc = CERA_CUDA_OK;
    for (uint32_t t = 0; t < max_col_tiles && rc == CERA_CUDA_OK; t += part) {
        TqParams q = p;
        const size_t first = (size_t)t * BN;
        q.col_tiles = max_col_tiles - t < part ? max_col_tiles - t : part;
        q.n = p.n - first < (size_t)q.col_tiles * BN ? (uint32_t)(p.n - first) : q.col_tiles * BN;
        q.out[0] = p.out[0] + first * p.ldc[0];
        rc = launch_tcq_part<T, BN>(q, ActView{x.scales + first * p.nb, x.quants + first * p.k, x.sums + first * (p.k / 16)}, scratch, st);
    }
    cudaFreeAsync(scratch, st);  // after the kernels above, in stream order
    return rc;
}

bool tcq_off() {
    static const bool v = [] {
        const char *e = getenv("CERA_CUDA_GEMM");
        return e && (strcmp(e, "mma") == 0 || strcmp(e, "columns") == 0);
    }();
    return v;
}

}  // namespace

bool gemm_tcq_supports(int type, size_t k) {
    if (tcq_off() || !is_block_type(type) || k == 0) return false;
    return k % (tq_kquant(type) ? 256 : 32) == 0;
}

// Fewer columns than this, and the kernels that need no operands in scratch are faster (device times of all launches, us, this
// kernel / the other).
//   Q8_0 and Q4_1, whose other kernel reads the weights once per eight columns.  4096 x 4096: 27 / 17 at 8 columns, 27 / 33 at 16, 92 /
//   1077 at 512; 2048 x 2048: 14 / 18 and 13 / 13 at 16; 2048 x 1024: 22 / 17 at 24, 22 / 22 at 32, 24 / 33 at 48; 1024 x 1024: 23 / 22 at 32,
//   13 / 33 at 48.
//   Q4_0 and Q6_K, whose other kernel is the mma.sync one, in tiles of 64 columns.  4096 x 4096: 23 / 16 at 32, 25 / 28 at 48, 26 / 30 at 64, 66 /
//   143 at 384; 2048 x 4096 and 4096 x 2048: 20 / 14 and 19 / 14 at 64, 22 / 24 and 22 / 27 at 96, 39 / 79 and 47 / 74 at 384; 2048 x 2048: 16 / 11 at
//   64, 18 / 20 at 96, 20 / 17 at 128, 23 / 33 at 160, 28 / 44 at 384; 1024 x 1024: 16 / 18 at 128 but 27 / 19 at 512 (Q6_K up to a tenth better
//   throughout).
static size_t tcq_min_columns(const WeightView &w) {
    const uint64_t weights = (uint64_t)w.m * w.k;
    switch (w.type) {
        case CERA_TYPE_Q4_1:
        case CERA_TYPE_Q8_0: return weights >= 1u << 22 ? 16 : 48;
        case CERA_TYPE_Q4_0:
        case CERA_TYPE_Q6_K: return weights >= 1u << 24 ? 48 : weights >= 1u << 23 ? 65 : weights >= 1u << 22 ? 129 : SIZE_MAX;
        default: return SIZE_MAX;  // Q4_K, Q5_K: gemm_tc.cu (14336 x 4096 x 512 without an image: 216 us, here 358)
    }
}

int32_t launch_gemm_tcq(const WeightView &w, const ActView &x, size_t n, float *out, size_t ldy, size_t ldc, int epilogue, cudaStream_t st, bool *taken) {
    *taken = false;
    if ((uintptr_t)x.quants % 16 || n < tcq_min_columns(w) || !gemm_tcq_supports(w.type, w.k)) return CERA_CUDA_OK;
    // A graph that is being captured stays one without allocation nodes, which may be cloned and nested: the other kernels need none.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return CERA_CUDA_OK;
    }
    TqParams p{};
    p.w[0] = w;
    p.out[0] = out;
    p.m[0] = w.m;
    p.ldc[0] = (uint32_t)ldc;
    p.n = (uint32_t)n;
    p.k = w.k;
    p.ldy = (uint32_t)ldy;
    p.epilogue = epilogue;
#define CERA_TCQ_PLAIN(BN, TILES)                                                                      \
    switch (w.type) {                                                                                  \
        case CERA_TYPE_Q4_0: return launch_tcq_bn<CERA_TYPE_Q4_0, BN>(p, 1, x, TILES, nullptr, st, taken); \
        case CERA_TYPE_Q4_1: return launch_tcq_bn<CERA_TYPE_Q4_1, BN>(p, 1, x, TILES, nullptr, st, taken); \
        case CERA_TYPE_Q8_0: return launch_tcq_bn<CERA_TYPE_Q8_0, BN>(p, 1, x, TILES, nullptr, st, taken); \
        default: return launch_tcq_bn<CERA_TYPE_Q6_K, BN>(p, 1, x, TILES, nullptr, st, taken);             \
    }
    if (n <= 32 && w.type != CERA_TYPE_Q4_0 && w.type != CERA_TYPE_Q6_K) {
        if (w.type == CERA_TYPE_Q4_1) return launch_tcq_bn<CERA_TYPE_Q4_1, 32>(p, 1, x, 1, nullptr, st, taken);
        return launch_tcq_bn<CERA_TYPE_Q8_0, 32>(p, 1, x, 1, nullptr, st, taken);
    }
    if (n <= 64) CERA_TCQ_PLAIN(64, 1)
    CERA_TCQ_PLAIN(128, (uint32_t)((n + 127) / 128))
#undef CERA_TCQ_PLAIN
}

size_t gemm_tcq_grouped_scratch(size_t k, uint32_t max_tiles) {
    return (size_t)max_tiles * TCQ_COLUMNS * ((k + TQ_KS - 1) / TQ_KS) * TQ_COL;
}

int32_t launch_gemm_tcq_grouped(const WeightView *ws, float *const *outs, int n_segs, const ActView &x, const MoeTile *tiles, const uint32_t *n_tiles,
                                uint32_t max_tiles, uint32_t rows_per_expert, size_t ldc, void *scratch_dev, cudaStream_t st) {
    if (!gemm_tcq_supports(ws[0].type, ws[0].k) || (uintptr_t)x.quants % 16 || max_tiles == 0 || n_segs < 1 || n_segs > 2 ||
        (n_segs == 2 && (ws[1].type != ws[0].type || ws[1].k != ws[0].k)))
        return fail(CERA_CUDA_ERR_STATE, "moe: a tensor-core plan without a tensor-core kernel");
    TqParams p{};
    for (int i = 0; i < n_segs; ++i) {
        p.w[i] = ws[i];
        p.out[i] = outs[i];
        p.m[i] = rows_per_expert;
        p.ldc[i] = (uint32_t)ldc;
    }
    p.k = ws[0].k;
    p.ldy = 1;
    p.epilogue = EPI_STORE;
    p.tiles = tiles;
    p.n_tiles = n_tiles;
    bool taken = false;
    CERA_DISPATCH_BLOCK_TYPE(ws[0].type, return (launch_tcq_bn<TT, 128>(p, n_segs, x, max_tiles, (uint8_t *)scratch_dev, st, &taken)));
    return CERA_CUDA_OK;
}

// bits 25..28: roles of the product over quantized bytes
static const bool g_tcq_status_registered = register_kernel_status([] {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_tcq_status, sizeof(v));
    return (uint32_t)v << 25;
});

}  // namespace cera

// Many-column bf16 products on the fifth-generation tensor cores: out[column][row] = W x, tcgen05.mma kind::f16 with f32
// accumulators in TMEM.  A persistent CTA walks output tiles of 128 weight rows x BN columns (tokens): one warp keeps a
// ring of stages filled by TMA (64 elements of k, 128-byte swizzle), one issues the MMAs, eight warps drain the
// finished accumulator - lane = weight row, so a column's values leave as consecutive stores; two warps share 32 rows and
// take 32 columns in turn - while the next tile's MMAs run into the other accumulator.
//
// In pairs (cta_group::2) two CTAs share tiles of 256 weight rows: each loads its 128 rows and half of the columns, and the tensor cores read both
// halves, which leaves shared memory half of the columns' traffic.  The even CTA's loader barrier counts both CTAs' bytes, its MMA warp issues for both.
//
// Grouped by expert the tiles come from a device-built work list.  With NA = 2 a stage holds two weight tiles (an expert's
// gate rows and the same up rows; without groups, the matrix's first and second half) against one activation tile, and the
// epilogue forms the gated unit from the two accumulators.  Every wait is bounded (tma.cuh); a wait that runs out empties the CTA and raises a status bit.
#include "dense.cuh"
#include "tc.cuh"
#include "tensor_map.h"

namespace cera {

__device__ unsigned int g_dense_tc_status = 0;

// bits 17..19: roles of this kernel (loader, MMA, epilogue); bits 20..22: the prompt attention's (attention_tc.cu)
static const bool g_dense_tc_registered = register_kernel_status([] {
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_dense_tc_status, sizeof(v));
    return (uint32_t)v << 17;
});

namespace {

constexpr int DT_BM = 128, DT_KS = 64, DT_THREADS = 10 * 32;  // loader, MMA, eight epilogue warps
constexpr uint32_t DT_A_BYTES = DT_BM * DT_KS * 2;

// PAIR: two CTAs on neighbouring SMs share a tile of 2 x 128 weight rows x BN columns: each holds its rows and half of the columns
template <int BN, int NA, bool PAIR>
struct Tile {
    static constexpr int ROWS = PAIR ? 2 * DT_BM : DT_BM, HALF = PAIR ? BN / 2 : BN;  // weight rows of a tile; columns a CTA loads
    static constexpr uint32_t B_BYTES = HALF * DT_KS * 2, STAGE = NA * DT_A_BYTES + B_BYTES;
    static constexpr int STAGES = 200 * 1024 / STAGE < 8 ? 200 * 1024 / STAGE : 8;
    static constexpr uint32_t ACC = NA * BN, COLS = 2 * ACC;  // TMEM columns of one accumulator, of both
    static constexpr uint32_t TMEM = COLS <= 64 ? 64 : COLS <= 128 ? 128 : COLS <= 256 ? 256 : 512;
    static constexpr uint32_t SMEM = STAGES * STAGE + 1024 + 256;
};

struct DtParams {
    DenseGemm g;
    uint32_t row_tiles, col_tiles;
};

// Output tile t of this launch.
struct DtTile {
    uint32_t a_row, row0, rows, first, end;
};
template <int BN, int NA, bool PAIR>
__device__ __forceinline__ DtTile dt_tile(const DtParams &p, uint32_t t) {
    constexpr uint32_t ROWS = Tile<BN, NA, PAIR>::ROWS;
    DtTile o;
    if (p.g.tiles) {
        const MoeTile m = p.g.tiles[t / p.row_tiles];
        o.row0 = (t % p.row_tiles) * ROWS;
        o.rows = NA == 2 ? p.g.rows_per_expert / 2 : p.g.rows_per_expert;
        o.a_row = m.expert * p.g.rows_per_expert + o.row0;
        o.first = m.first;
        o.end = m.first + m.count;
    } else {
        o.row0 = o.a_row = (t / p.col_tiles) * ROWS;
        o.rows = p.g.w.rows / NA;
        o.first = (t % p.col_tiles) * BN;
        o.end = min(o.first + BN, p.g.n);
    }
    return o;
}

template <int BN, int NA, bool PAIR>
__global__ void __launch_bounds__(DT_THREADS, 1) dense_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, DtParams p) {
    using S = Tile<BN, NA, PAIR>;
    extern __shared__ uint8_t raw[];
    uint8_t *stages = raw + (1024 - (tma::smem_u32(raw) & 1023)) % 1024;
    uint64_t *full = reinterpret_cast<uint64_t *>(stages + S::STAGES * S::STAGE), *empty = full + S::STAGES, *acc_full = empty + S::STAGES, *acc_empty = acc_full + 2;
    uint32_t *tmem_at = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile uint32_t *abort_flag = tmem_at + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? blockIdx.x & 1 : 0, first_tile = PAIR ? blockIdx.x / 2 : blockIdx.x, step = PAIR ? gridDim.x / 2 : gridDim.x;
    pdl_trigger();
    if (threadIdx.x == 0) {
        for (int i = 0; i < S::STAGES; ++i) {
            tma::mbar_init(full + i, 1);
            tma::mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            tma::mbar_init(acc_full + i, 1);
            tma::mbar_init(acc_empty + i, PAIR ? 16 : 8);  // the epilogue warps; the even CTA's barrier counts both CTAs'
        }
        *abort_flag = 0;
        tma::mbar_init_fence();
    }
    __syncwarp();
    // A pair allocates for both of its SMs: both CTAs run by then, and have what they asked for before either goes on.
    if constexpr (PAIR) cluster_barrier();
    if (warp == 1) {
        if constexpr (PAIR) {
            tmem_alloc_pair(tmem_at, S::TMEM);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(tmem_at, S::TMEM);
            tmem_relinquish();
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_barrier();  // (the barriers of both CTAs are there, too)
    tc_fence_after();
    const uint32_t tmem = *tmem_at;
    pdl_wait();
    const uint32_t n_tiles = p.g.tiles ? *p.g.n_tiles * p.row_tiles : p.row_tiles * p.col_tiles, n_k = p.g.w.ld / DT_KS;
    // a ragged tile's products stop at its last column (in whole 32s, as the epilogue reads them): an expert's last item.
    // 2048 tokens through four layers of routed experts at width 4096: 4.50 -> 4.42 ms, 1.4 to 2.4 % in three pairs of runs that
    // repeat within 1 %
    auto columns = [](const DtTile &o) { return min((uint32_t)BN, (o.end - o.first + 31) & ~31u); };
    if (warp == 0) {  // the whole warp, one lane requests
        const uint32_t me = elect_one();
        uint32_t it = 0;
        bool ok = true;
        for (uint32_t t = first_tile; t < n_tiles && ok; t += step) {
            const DtTile o = dt_tile<BN, NA, PAIR>(p, t);
            const uint32_t x0 = p.g.block_rows ? o.a_row / p.g.block_rows * p.g.w.ld : 0;
            const uint32_t a_row = o.a_row + rank * DT_BM, col = o.first + rank * (columns(o) / 2);
            for (uint32_t k = 0; k < n_k; ++k, ++it) {
                const uint32_t s = it % S::STAGES;
                if (!(ok = tma::mbar_wait_warp(empty + s, (it / S::STAGES & 1) ^ 1, abort_flag, &g_dense_tc_status, 1u))) break;
                uint8_t *st = stages + s * S::STAGE;
                if constexpr (PAIR) {  // all bytes of both CTAs are counted on the even CTA's barrier
                    tma::mbar_expect_tx_if(full + s, 2 * S::STAGE, rank == 0 ? me : 0);
                    const uint32_t bar = tma::smem_of_rank(full + s, 0);
                    tma::tensor_g2s_2d_pair_if(st, &map_w, k * DT_KS, a_row, bar, me);
                    if (NA == 2) tma::tensor_g2s_2d_pair_if(st + DT_A_BYTES, &map_w, k * DT_KS, a_row + o.rows, bar, me);
                    tma::tensor_g2s_2d_pair_if(st + NA * DT_A_BYTES, &map_x, x0 + k * DT_KS, col, bar, me);
                } else {
                    tma::mbar_expect_tx_if(full + s, S::STAGE, me);
                    tma::tensor_g2s_2d_if(st, &map_w, k * DT_KS, o.a_row, full + s, me);
                    if (NA == 2) tma::tensor_g2s_2d_if(st + DT_A_BYTES, &map_w, k * DT_KS, o.a_row + o.rows, full + s, me);
                    tma::tensor_g2s_2d_if(st + NA * DT_A_BYTES, &map_x, x0 + k * DT_KS, o.first, full + s, me);
                }
            }
        }
        // This CTA's shared memory must outlive the copies in flight (they only are when something gave up) and, of a pair, the last products'
        // arrivals on its barriers: what those wait for includes its copies.
        if (PAIR || *abort_flag) {
            uint64_t *last = PAIR ? empty : full;
            for (uint32_t i = it > S::STAGES ? it - S::STAGES : 0; i < it; ++i)
                for (uint32_t n = 0; n < tma::SPIN_LIMIT && !tma::mbar_test(last + i % S::STAGES, i / S::STAGES & 1); ++n) __nanosleep(40);
        }
    } else if (warp == 1) {
        if (rank == 0) {  // the whole warp, one lane issues
            const uint32_t me = elect_one();
            uint32_t it = 0, j = 0;
            bool ok = true;
            auto arrived = [&](uint64_t *bar, uint32_t parity) {
                return tma::mbar_wait_warp(bar, parity, abort_flag, &g_dense_tc_status, 2u);
            };
            for (uint32_t t = first_tile; t < n_tiles && ok; t += step, ++j) {
                const uint32_t b = j & 1, acc = tmem + b * S::ACC;
                const DtTile o = dt_tile<BN, NA, PAIR>(p, t);
                const uint32_t idesc = tc_idesc_bf16(S::ROWS, columns(o));
                if (!(ok = arrived(acc_empty + b, (j >> 1 & 1) ^ 1))) break;
                tc_fence_after();
                for (uint32_t k = 0; k < n_k; ++k, ++it) {
                    const uint32_t s = it % S::STAGES;
                    if (!(ok = arrived(full + s, it / S::STAGES & 1))) break;
                    tc_fence_after();
                    const uint32_t st = tma::smem_u32(stages + s * S::STAGE);
                    const uint64_t da = smem_desc_sw128(st), da2 = smem_desc_sw128(st + DT_A_BYTES), db = smem_desc_sw128(st + NA * DT_A_BYTES);
#pragma unroll
                    for (int kk = 0; kk < DT_KS / 16; ++kk)
#pragma unroll
                        for (int a = 0; a < NA; ++a) {
                            if constexpr (PAIR) tc_mma_f16_pair(acc + a * BN, (a ? da2 : da) + 2 * kk, db + 2 * kk, idesc, k | kk, me);
                            else tc_mma_f16(acc + a * BN, (a ? da2 : da) + 2 * kk, db + 2 * kk, idesc, k | kk, me);
                        }
                    if constexpr (PAIR) tc_commit_pair(empty + s, me);
                    else tc_commit(empty + s, me);
                }
                if (!ok) break;
                if constexpr (PAIR) tc_commit_pair(acc_full + b, me);
                else tc_commit(acc_full + b, me);
            }
        }
    } else {
        const uint32_t quad = warp & 3;  // the TMEM lanes this warp may read: [32 quad, + 32)
        const uint32_t turn = (warp - 2) >> 2;
        uint32_t j = 0;
        for (uint32_t t = first_tile; t < n_tiles; t += step, ++j) {
            const uint32_t b = j & 1;
            if (!tma::mbar_wait_warp(acc_full + b, j >> 1 & 1, abort_flag, &g_dense_tc_status, 4u)) break;
            tc_fence_after();
            const DtTile o = dt_tile<BN, NA, PAIR>(p, t);
            const uint32_t row = o.row0 + rank * DT_BM + quad * 32 + lane, acc = tmem + b * S::ACC + (quad * 32 << 16), cols = o.end - o.first;
            const bool live = row < o.rows;
#pragma unroll 1
            for (uint32_t c0 = turn * 32; c0 < BN && c0 < cols; c0 += 64) {
                uint32_t v[2][16];
                tmem_ld16(acc + c0, v[0]);
                tmem_ld16(acc + c0 + 16, v[1]);
                if (NA == 2) {
                    uint32_t u[2][16];
                    tmem_ld16(acc + BN + c0, u[0]);
                    tmem_ld16(acc + BN + c0 + 16, u[1]);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        const uint32_t col = o.first + c0 + c;
                        if (live && col < o.end) {
                            const float sc = p.g.col_scale ? p.g.col_scale[col] : 1.0f;
                            ((bf16 *)p.g.out)[(size_t)col * p.g.ldo + row] = __float2bfloat16_rn(
                                gated_unit(sc * __uint_as_float(v[c >> 4][c & 15]), sc * __uint_as_float(u[c >> 4][c & 15]), p.g.act));
                        }
                    }
                    continue;
                }
                tmem_wait_ld();
                if (p.g.out_kind == DENSE_F32) {
                    float *out = (float *)p.g.out + (size_t)(o.first + c0) * p.g.ldo + row;
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (live && c0 + c < cols) out[(size_t)c * p.g.ldo] = __uint_as_float(v[c >> 4][c & 15]);
                } else if (p.g.out_kind == DENSE_T) {
                    bf16 *out = (bf16 *)p.g.out + (size_t)(o.first + c0) * p.g.ldo + row;
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (live && c0 + c < cols) out[(size_t)c * p.g.ldo] = __float2bfloat16_rn(__uint_as_float(v[c >> 4][c & 15]));
                } else if (live) {  // transposed: 32 consecutive columns of this row; columns past the end are zeros of the operand
                    uint4 *out = reinterpret_cast<uint4 *>((bf16 *)p.g.out + (size_t)row * p.g.ldo + o.first + c0);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int c = q * 8 + i * 2;
                            const __nv_bfloat162 pr = __floats2bfloat162_rn(__uint_as_float(v[c >> 4][c & 15]), __uint_as_float(v[c >> 4][(c & 15) + 1]));
                            w[i] = *reinterpret_cast<const uint32_t *>(&pr);
                        }
                        if (o.first + c0 + q * 8 + 8 <= p.g.ldo) out[q] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            tc_fence_before();
            if (lane == 0) {
                if constexpr (PAIR) tma::mbar_arrive_cluster(tma::smem_of_rank(acc_empty + b, 0));
                else tma::mbar_arrive(acc_empty + b);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) {
        cluster_barrier();  // the other CTA's products read this one's shared memory, its warps arrive here
        if (warp == 1) tmem_dealloc_pair(tmem, S::TMEM);
        __syncwarp();
        cluster_barrier();  // neither leaves before both have given back
    } else {
        if (warp == 1) tmem_dealloc(tmem, S::TMEM);
    }
}

template <int BN, int NA, bool PAIR = false>
int32_t launch_tc(const DenseGemm &g, cudaStream_t st) {
    using S = Tile<BN, NA, PAIR>;
    CUtensorMap mw, mx;
    CERA_TRY(tensor_map_bf16(&mw, g.w.w, g.w.rows, g.w.ld, DT_KS, DT_BM));
    CERA_TRY(tensor_map_bf16(&mx, g.x, g.n, g.row_len(), DT_KS, S::HALF));
    DtParams p;
    p.g = g;
    const uint32_t rows = (g.tiles ? g.rows_per_expert : g.w.rows) / NA;
    p.row_tiles = (rows + S::ROWS - 1) / S::ROWS;
    p.col_tiles = g.tiles ? g.max_tiles : (g.n + BN - 1) / BN;
    const uint64_t tiles = (uint64_t)p.row_tiles * p.col_tiles, room = (uint64_t)sm_count() / (PAIR ? 2 : 1);
    const unsigned grid = (unsigned)(tiles < room ? tiles : room);
    auto k = dense_gemm_tc_kernel<BN, NA, PAIR>;
    CERA_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
    count_launch();
    if (PAIR) return check_cuda(launch_pairs(k, grid, dim3(DT_THREADS), S::SMEM, st, mw, mx, p), "dense tcgen05 gemm (pairs) launch");
    return check_cuda(launch_k(k, dim3(grid), dim3(DT_THREADS), S::SMEM, st, mw, mx, p), "dense tcgen05 gemm launch");
}

}  // namespace

int32_t launch_dense_gemm_tc(const DenseGemm &g, cudaStream_t st, bool *taken) {
    *taken = false;
    if (g.w.f32 || g.w.ld % DT_KS || g.n == 0) return CERA_CUDA_OK;
    if (g.out_kind == DENSE_T_TRANSPOSED && g.ldo % 8) return CERA_CUDA_OK;
    *taken = true;
    const bool unit = g.out_kind == DENSE_GATED_UNIT;
    // A pair of CTAs per tile where a tile has more than 64 columns - of experts, where they fill it on average: 52 columns an expert, width 2048, 60.5 us
    // alone and 61.4 in pairs, 64 60.7 and 61.3, 96 67.9 and 67.0, 128 70.9 and 70.1 (width 4096 218 and 211), whole prompts even at 128 - unless the last pair of
    // row tiles would leave more than an eighth of the work for rows that are not there.  2048 tokens at
    // width 4096, single CTAs and pairs: four layers of experts 4.22 and 4.05 ms, eight dense layers 6.65 and 6.36; 200 tokens through a gated unit 43.2
    // and 41.0 us (at up to 64 columns the weights are read once either way).
    const uint32_t rows = (g.tiles ? g.rows_per_expert : g.w.rows) / (unit ? 2 : 1), whole = (rows + DT_BM - 1) / DT_BM;
    const bool full = !g.tiles || g.n >= g.w.rows / g.rows_per_expert * DT_BM;
    const bool two = full && (whole + 1) / 2 * 16 <= whole * 9 && g.block_rows % (2 * DT_BM) == 0;
    if (g.tiles) {
        if (g.group_columns <= 32) return unit ? launch_tc<32, 2>(g, st) : launch_tc<32, 1>(g, st);
        if (g.group_columns <= 64) return unit ? launch_tc<64, 2>(g, st) : launch_tc<64, 1>(g, st);
        if (two) return unit ? launch_tc<128, 2, true>(g, st) : launch_tc<128, 1, true>(g, st);
        return unit ? launch_tc<128, 2>(g, st) : launch_tc<128, 1>(g, st);
    }
    if (unit) {
        if (two && g.n > 64) return launch_tc<128, 2, true>(g, st);
        return g.n <= 32 ? launch_tc<32, 2>(g, st) : g.n <= 64 ? launch_tc<64, 2>(g, st) : launch_tc<128, 2>(g, st);
    }
    const uint32_t row_tiles = (g.w.rows + DT_BM - 1) / DT_BM;
    if (g.n <= 32) return launch_tc<32, 1>(g, st);
    if (g.n <= 64) return launch_tc<64, 1>(g, st);
    if (g.n <= 128 || row_tiles * ((g.n + 255) / 256) < (uint32_t)sm_count() * 3 / 4) return launch_tc<128, 1>(g, st);
    if (two) return launch_tc<256, 1, true>(g, st);
    return launch_tc<256, 1>(g, st);
}

}  // namespace cera

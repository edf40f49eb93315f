// W4A4 (H256, g64) GEMM on byte-wide (E4M3) codes for few rows or outputs: one tile per CTA, 128 rows x 64 or 32 outputs,
// or (EXCHANGED) 128 outputs x 16, 32 or 48 rows. Same
// operator, arithmetic and bits as w4a4_pair_gemm.cuh (reference: qwen_image_cuda/cuda/gemm.cu:65-189).
//
// The groups of an output are added in order, so K cannot be split, and a tile is a chain of k / 256 hand-overs from the
// tensor cores to the fold warps, of four groups each. With few rows, tiles of 256 leave most SMs idle or folding zeros; here 77 x 9216 outputs are
// 144 tiles. What counts is the length of the chain's links:
//   * a TMEM buffer holds four groups, one stage of 256 inputs: one commit, one look and one hand-back per four groups
//   * two issuing warps take the stages in turn (an issuing warp needs some 500 cycles per turn)
//   * a fold warp copies the next group's dots out of TMEM while it folds the current one
//
// EXCHANGED, the weights are the 128 rows and 16 to 48 activation rows the columns: nothing is folded for rows that do not
// exist, and a lane, which owns an output, writes next to its neighbours (77 x 9216 x 3072 11.7 -> 10.4 us, 16 rows 11.3 -> 8.4).
// What bounds it then: 16 columns still take 0.073 us a group (0.11 where rows lie a multiple of 4096 bytes apart), half of that
// the 32 KB of weights a stage coming into the SM.
//
//   warp 0      TMA: A rows (only those that exist, rounded up to 16) and B rows, 256 inputs a stage
//   warps 1, 3  tcgen05.mma kind::f8f6f4, M = 128, N = the tile's columns
//   warp 2      weight scales to fp32 in shared memory
//   warps 4-19  fold: 32 rows x a quarter of the columns each; a thread owns a row and reads its scales itself
#pragma once
#include "ptx.cuh"
#include "w4a16_gemm.cuh"
#include "w4a4_pair_gemm.cuh"

namespace qi {
namespace w4a4_narrow {

using w4a4_pair::lds_pairs;

constexpr int BM = 128, STAGE_K = 256, STAGE_GROUPS = 4, K_HALVES = STAGE_K / 128;
constexpr int PRODUCER_WARP = 0, MMA_WARP = 1, SCALE_WARP = 2, SECOND_MMA_WARP = 3, FOLD_WARP0 = 4, FOLD_WARPS = 16;
constexpr int THREADS = 32 * (FOLD_WARP0 + FOLD_WARPS);
constexpr int ISSUERS = 2, STAGES = 4, SLOTS = 4;  // SLOTS: stages of weight scales
constexpr uint32_t AHEAD_BACKOFF_NS = 100, FOLD_BACKOFF_NS = 20;

template <int BN>
struct Tile {
    static constexpr int COLUMNS = BN / 4;  // of a fold warp
    static constexpr int A_HALF_BYTES = BM * 128, B_HALF_BYTES = BN * 128;
    static constexpr int A_BYTES = K_HALVES * A_HALF_BYTES, B_BYTES = K_HALVES * B_HALF_BYTES;
    static constexpr int SW_BYTES = STAGE_GROUPS * BN * 4;
    static constexpr int BUFFERS = BN <= 32 ? 4 : 2;
    static constexpr int BUFFER_COLUMNS = STAGE_GROUPS * BN, TMEM_COLUMNS = BUFFERS * BUFFER_COLUMNS > 256 ? 512 : 256;
    static constexpr int BARRIER_BYTES = 256;
    static constexpr int SMEM_BYTES = STAGES * (A_BYTES + B_BYTES) + SLOTS * SW_BYTES + BARRIER_BYTES + 1024;
    static_assert(SMEM_BYTES <= 232448 && SMEM_BYTES >= ONE_CTA_SMEM, "one CTA per SM: a second would wait for TMEM");
    static_assert(BUFFERS * BUFFER_COLUMNS <= TMEM_COLUMNS, "TMEM allocation size");
    static_assert((2 * STAGES + 2 * SLOTS + 2 * BUFFERS) * 8 + 4 <= BARRIER_BYTES, "barrier block");
};

// 32 TMEM lanes x N columns into N / 2 64-bit registers, and the wait for them with the registers tied to it.
template <int N>
__device__ __forceinline__ void load_dots(uint32_t address, uint64_t (&r)[N / 2]) {
    if constexpr (N == 16) {
        asm volatile(
            "{\n\t.reg .b32 t<16>;\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {t0, t1, t2, t3, t4, t5, t6, t7, t8, t9, t10, t11, t12, t13, t14, t15}, [%8];\n\t"
            "mov.b64 %0, {t0, t1};\n\tmov.b64 %1, {t2, t3};\n\tmov.b64 %2, {t4, t5};\n\tmov.b64 %3, {t6, t7};\n\t"
            "mov.b64 %4, {t8, t9};\n\tmov.b64 %5, {t10, t11};\n\tmov.b64 %6, {t12, t13};\n\tmov.b64 %7, {t14, t15};\n\t}"
            : "=l"(r[0]), "=l"(r[1]), "=l"(r[2]), "=l"(r[3]), "=l"(r[4]), "=l"(r[5]), "=l"(r[6]), "=l"(r[7])
            : "r"(address)
            : "memory");
    } else {
        static_assert(N == 4 || N == 8 || N == 12, "4, 8, 12 or 16 columns");
        if constexpr (N >= 8)
            asm volatile(
                "{\n\t.reg .b32 t<8>;\n\t"
                "tcgen05.ld.sync.aligned.32x32b.x8.b32 {t0, t1, t2, t3, t4, t5, t6, t7}, [%4];\n\t"
                "mov.b64 %0, {t0, t1};\n\tmov.b64 %1, {t2, t3};\n\tmov.b64 %2, {t4, t5};\n\tmov.b64 %3, {t6, t7};\n\t}"
                : "=l"(r[0]), "=l"(r[1]), "=l"(r[2]), "=l"(r[3])
                : "r"(address)
                : "memory");
        if constexpr (N != 8)
            asm volatile(
                "{\n\t.reg .b32 t<4>;\n\t"
                "tcgen05.ld.sync.aligned.32x32b.x4.b32 {t0, t1, t2, t3}, [%2];\n\t"
                "mov.b64 %0, {t0, t1};\n\tmov.b64 %1, {t2, t3};\n\t}"
                : "=l"(r[N / 2 - 2]), "=l"(r[N / 2 - 1])
                : "r"(address + N - 4)
                : "memory");
    }
}
template <int N>
__device__ __forceinline__ void wait_dots(uint64_t (&r)[N / 2]) {
    if constexpr (N == 16)
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+l"(r[0]), "+l"(r[1]), "+l"(r[2]), "+l"(r[3]), "+l"(r[4]), "+l"(r[5]), "+l"(r[6]), "+l"(r[7])::"memory");
    else if constexpr (N == 12)
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+l"(r[0]), "+l"(r[1]), "+l"(r[2]), "+l"(r[3]), "+l"(r[4]), "+l"(r[5])::"memory");
    else if constexpr (N == 8)
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+l"(r[0]), "+l"(r[1]), "+l"(r[2]), "+l"(r[3])::"memory");
    else
        asm volatile("tcgen05.wait::ld.sync.aligned;" : "+l"(r[0]), "+l"(r[1])::"memory");
}

// EXCHANGED: the 128 rows of a tile are outputs (weight rows), its columns activation rows; map_a and a_scales then are
// the weights'. dot * sw and sw * sa are as exact as dot * sa and sa * sw: the same bits.
template <int BN, bool EXCHANGED>
__global__ void __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
            const __half *__restrict__ a_scales, const __half *__restrict__ w_scales,
            const float *__restrict__ bias, void *__restrict__ y, const GemmShape shape, const int a_box_rows) {
    using T = Tile<BN>;
    constexpr int COLUMNS = T::COLUMNS, BUFFERS = T::BUFFERS;
    static_assert(EXCHANGED || COLUMNS % 8 == 0, "a thread stores its columns 16 bytes at a time");
    const int rows_of_a = EXCHANGED ? shape.n : shape.m, rows_of_w = EXCHANGED ? shape.m : shape.n;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float *sw_slots = reinterpret_cast<float *>(smem + STAGES * (T::A_BYTES + T::B_BYTES));
    uint64_t *barriers = reinterpret_cast<uint64_t *>(sw_slots + SLOTS * STAGE_GROUPS * BN);
    const uint32_t tile_a = smem_u32(smem), tile_b = tile_a + STAGES * T::A_BYTES, sw_tile = smem_u32(sw_slots);
    const uint32_t full = smem_u32(barriers), empty = full + 8 * STAGES, sw_full = empty + 8 * STAGES, sw_empty = sw_full + 8 * SLOTS;
    const uint32_t dot_full = sw_empty + 8 * SLOTS, dot_empty = dot_full + 8 * BUFFERS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(barriers + 2 * STAGES + 2 * SLOTS + 2 * BUFFERS);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int tiles_m = (rows_of_a + BM - 1) / BM, tiles_n = (rows_of_w + BN - 1) / BN, tiles = tiles_m * tiles_n;
    const int k_stages = shape.k / STAGE_K, groups = shape.k / 64;
    const int my_tiles = static_cast<int>(blockIdx.x) < tiles ? (tiles - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;
    const uint32_t total = static_cast<uint32_t>(my_tiles) * k_stages;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbarrier_init(barriers + s, 1);
            mbarrier_init(barriers + STAGES + s, 1);
        }
        for (int s = 0; s < SLOTS; ++s) {
            mbarrier_init(barriers + 2 * STAGES + s, 1);
            mbarrier_init(barriers + 2 * STAGES + SLOTS + s, FOLD_WARPS);
        }
        for (int b = 0; b < BUFFERS; ++b) {
            mbarrier_init(barriers + 2 * STAGES + 2 * SLOTS + b, 1);
            mbarrier_init(barriers + 2 * STAGES + 2 * SLOTS + BUFFERS + b, FOLD_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == PRODUCER_WARP && elect_one()) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_w);
    }
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, T::TMEM_COLUMNS);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    grid_wait();
    grid_release();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == PRODUCER_WARP) {
        uint32_t s = 0, phase = 1;
        bool alive = true;
        for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x) {
            const int m0 = tile % tiles_m * BM, n0 = tile / tiles_m * BN;
            for (int ks = 0; ks < k_stages; ++ks) {
                if (!mbarrier_wait_uniform(empty + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0x9000 | s, AHEAD_BACKOFF_NS)) { alive = false; break; }
                if (elect_one()) {
                    mbarrier_arrive_expect_tx_u32(full + s * 8, K_HALVES * (a_box_rows * 128 + T::B_HALF_BYTES));
#pragma unroll
                    for (int half = 0; half < K_HALVES; ++half) {
                        tma_load_2d_u32(tile_a + s * T::A_BYTES + half * T::A_HALF_BYTES, &map_a, full + s * 8, ks * STAGE_K + half * 128, m0);
                        tma_load_2d_u32(tile_b + s * T::B_BYTES + half * T::B_HALF_BYTES, &map_w, full + s * 8, ks * STAGE_K + half * 128, n0);
                    }
                }
                __syncwarp();
                if (++s == STAGES) s = 0, phase ^= 1;
            }
        }
    } else if (warp == MMA_WARP || warp == SECOND_MMA_WARP) {
        constexpr uint32_t idesc = umma_idesc_e4m3_f32(BM, BN);
        static_assert(BUFFERS % ISSUERS == 0 && STAGES % ISSUERS == 0, "a warp keeps to every other buffer and stage");
        const uint32_t mine = warp == MMA_WARP ? 0 : 1;
        const uint64_t a_first = umma_desc_k_sw128(tile_a), b_first = umma_desc_k_sw128(tile_b);
        uint32_t s = mine, phase = 0, buffer = mine, buffer_phase = 1;
        for (uint32_t stage = mine; stage < total; stage += ISSUERS) {
            if (!mbarrier_wait_uniform2(full + s * 8, phase, dot_empty + buffer * 8, buffer_phase, &g_status, STATUS_WAIT_TMEM_EMPTY | 0x9000 | s)) break;
            tcgen05_fence_after();
            if (elect_one()) {
                const uint32_t accumulator = tmem_base + buffer * T::BUFFER_COLUMNS;
                const uint64_t a_desc = a_first + s * (T::A_BYTES >> 4), b_desc = b_first + s * (T::B_BYTES >> 4);
#pragma unroll
                for (int g = 0; g < STAGE_GROUPS; ++g)
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk)
                        umma_f8(accumulator + g * BN, a_desc + (g >> 1) * (T::A_HALF_BYTES >> 4) + (g & 1) * 4 + kk * 2,
                                b_desc + (g >> 1) * (T::B_HALF_BYTES >> 4) + (g & 1) * 4 + kk * 2, idesc, kk);
                tcgen05_commit_u32(dot_full + buffer * 8);
                tcgen05_commit_u32(empty + s * 8);
            }
            __syncwarp();
            buffer += ISSUERS;
            if (buffer >= BUFFERS) buffer -= BUFFERS, buffer_phase ^= 1;
            s += ISSUERS;
            if (s >= STAGES) s -= STAGES, phase ^= 1;
        }
    } else if (warp == SCALE_WARP) {
        // four groups' scales (eight bytes) of up to two columns per lane, loaded one stage ahead
        constexpr int ITEMS = (BN + 31) / 32;
        uint32_t slot = 0, phase = 1;
        bool alive = true;
        for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x) {
            const int n0 = tile / tiles_m * BN;
            const __half *rows[ITEMS];
            uint2 next[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const int column = n0 + i * 32 + lane < rows_of_w ? n0 + i * 32 + lane : rows_of_w - 1;
                rows[i] = w_scales + static_cast<size_t>(column) * groups;
                next[i] = __ldg(reinterpret_cast<const uint2 *>(rows[i]));
            }
            for (int ks = 0; ks < k_stages; ++ks) {
                uint2 now[ITEMS];
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    now[i] = next[i];
                    if (ks + 1 < k_stages) next[i] = __ldg(reinterpret_cast<const uint2 *>(rows[i]) + ks + 1);
                }
                if (!mbarrier_wait_uniform(sw_empty + slot * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0x9100 | slot, AHEAD_BACKOFF_NS)) { alive = false; break; }
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    if (BN % 32 != 0 && i * 32 + lane >= BN) break;
                    const float2 low = __half22float2(*reinterpret_cast<const __half2 *>(&now[i].x)), high = __half22float2(*reinterpret_cast<const __half2 *>(&now[i].y));
                    float *to = sw_slots + slot * (STAGE_GROUPS * BN) + i * 32 + lane;
                    to[0] = low.x, to[BN] = low.y, to[2 * BN] = high.x, to[3 * BN] = high.y;
                }
                __syncwarp();
                if (lane == 0) mbarrier_arrive_u32(sw_full + slot * 8);
                if (++slot == SLOTS) slot = 0, phase ^= 1;
            }
        }
    } else {
        const int quadrant = warp & 3, slice = (warp - FOLD_WARP0) >> 2;
        const uint32_t tmem_lane = tmem_base + slice * COLUMNS + (static_cast<uint32_t>(quadrant * 32) << 16);
        uint32_t buffer = 0, buffer_phase = 0, slot = 0, slot_phase = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < tiles && alive; tile += gridDim.x) {
            const int first_row = tile % tiles_m * BM + quadrant * 32, row = first_row + lane, n0 = tile / tiles_m * BN + slice * COLUMNS;
            const bool busy = first_row < rows_of_a && n0 < rows_of_w;  // a warp without outputs only hands the buffers back
            const uint2 *row_scales = reinterpret_cast<const uint2 *>(a_scales + static_cast<size_t>(row < rows_of_a ? row : rows_of_a - 1) * groups);
            uint2 sa_next = busy ? __ldg(row_scales) : make_uint2(0u, 0u);
            const float add = EXCHANGED && bias != nullptr && busy && row < rows_of_a ? __ldg(bias + row) : 0.0f;  // long there when it is asked for
            uint64_t acc[COLUMNS / 2];
#pragma unroll
            for (int j = 0; j < COLUMNS / 2; ++j) acc[j] = 0;
#pragma unroll 1
            for (int ks = 0; ks < k_stages; ++ks) {
                const float2 sa_low = __half22float2(*reinterpret_cast<const __half2 *>(&sa_next.x)), sa_high = __half22float2(*reinterpret_cast<const __half2 *>(&sa_next.y));
                const float sa[STAGE_GROUPS] = {sa_low.x, sa_low.y, sa_high.x, sa_high.y};
                if (busy && ks + 1 < k_stages) sa_next = __ldg(row_scales + ks + 1);
                if (!mbarrier_wait_uniform2(dot_full + buffer * 8, buffer_phase, sw_full + slot * 8, slot_phase, &g_status, STATUS_WAIT_TMEM_FULL | 0x9000 | buffer,
                                            FOLD_BACKOFF_NS)) { alive = false; break; }
                tcgen05_fence_after();
                if (busy) {
                    const uint32_t tmem = tmem_lane + buffer * T::BUFFER_COLUMNS, sw = sw_tile + slot * T::SW_BYTES + slice * COLUMNS * 4;
                    uint64_t dots[2][COLUMNS / 2];
                    load_dots<COLUMNS>(tmem, dots[0]);
#pragma unroll
                    for (int g = 0; g < STAGE_GROUPS; ++g) {
                        const uint64_t sa2 = pack_f32x2(sa[g], sa[g]);
                        ulonglong2 sw4[COLUMNS / 4];
#pragma unroll
                        for (int q = 0; q < COLUMNS / 4; ++q) sw4[q] = lds_pairs(sw + (g * BN + 4 * q) * 4);
                        wait_dots<COLUMNS>(dots[g & 1]);
                        if (g + 1 < STAGE_GROUPS) {
                            load_dots<COLUMNS>(tmem + (g + 1) * BN, dots[(g + 1) & 1]);
                        } else {
                            tcgen05_fence_before();
                            __syncwarp();
                            if (lane == 0) mbarrier_arrive_u32(dot_empty + buffer * 8);
                        }
#pragma unroll
                        for (int q = 0; q < COLUMNS / 4; ++q) {  // dot * sa and sa * sw are exact: rounded once, in the fused multiply-add
                            acc[2 * q] = fma_f32x2(mul_f32x2(dots[g & 1][2 * q], sa2), sw4[q].x, acc[2 * q]);
                            acc[2 * q + 1] = fma_f32x2(mul_f32x2(dots[g & 1][2 * q + 1], sa2), sw4[q].y, acc[2 * q + 1]);
                        }
                    }
                } else {
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbarrier_arrive_u32(dot_empty + buffer * 8);
                }
                __syncwarp();
                if (lane == 0) mbarrier_arrive_u32(sw_empty + slot * 8);
                if (++buffer == BUFFERS) buffer = 0, buffer_phase ^= 1;
                if (++slot == SLOTS) slot = 0, slot_phase ^= 1;
            }
            if (!alive || !busy || row >= rows_of_a) continue;
            float out[COLUMNS];
#pragma unroll
            for (int j = 0; j < COLUMNS / 2; ++j) unpack_f32x2(acc[j], out[2 * j], out[2 * j + 1]);
            if constexpr (EXCHANGED) {  // a lane owns an output: a warp writes 32 of an activation row at a time
#pragma unroll
                for (int j = 0; j < COLUMNS; ++j) {
                    if (n0 + j >= shape.m) break;
                    const size_t element = static_cast<size_t>(n0 + j) * shape.ldy + row;
                    const float value = bias != nullptr ? out[j] + add : out[j];
                    if (shape.y_is_half) static_cast<__half *>(y)[element] = __float2half_rn(value);
                    else static_cast<float *>(y)[element] = value;
                }
                continue;
            }
            if (bias != nullptr) {
#pragma unroll
                for (int j = 0; j < COLUMNS; ++j) out[j] += __ldg(bias + n0 + j);  // n is a multiple of 32: the columns all exist
            }
            const size_t element = static_cast<size_t>(row) * shape.ldy + n0;
            if (shape.y_is_half) {
#pragma unroll
                for (int j = 0; j < COLUMNS; j += 8) {
                    uint32_t h[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const __half2 pair = __floats2half2_rn(out[j + 2 * i], out[j + 2 * i + 1]);
                        h[i] = *reinterpret_cast<const uint32_t *>(&pair);
                    }
                    *reinterpret_cast<uint4 *>(static_cast<__half *>(y) + element + j) = make_uint4(h[0], h[1], h[2], h[3]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < COLUMNS; j += 4)
                    *reinterpret_cast<float4 *>(static_cast<float *>(y) + element + j) = make_float4(out[j], out[j + 1], out[j + 2], out[j + 3]);
            }
        }
        tmem_load_wait();
    }

    tcgen05_fence_before();
    __syncthreads();
    if (*reinterpret_cast<volatile uint32_t *>(&g_status) != 0) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let bulk copies already issued land
    }
    if (warp == MMA_WARP) {
        __syncwarp();
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, T::TMEM_COLUMNS);
    }
}

}  // namespace w4a4_narrow
}  // namespace qi

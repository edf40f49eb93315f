// W4A16 g64 dequant-GEMM on pairs of CTAs with the operands' roles exchanged, for many activation rows: 256 weight rows
// (128 per CTA, unpacked straight into TMEM) x up to 256 activation rows per tile. Same operator and unpacking as
// w4a16_gemm.cuh (reference: qwen_image_cuda/cuda/gemm.cu:191-268), same exchange as w4a16_swap_gemm.cuh.
//
// A large GEMM runs into the power limit, not into a pipe (SM clocks near 1.4 of 1.965 GHz), so what a tile moves through
// shared memory counts twice. With the weights as the SECOND operand every unpacked weight is written to shared memory
// and read back by the tensor cores, beside the activations: 88 KB per 64 inputs and CTA. Here the weights go from
// registers into TMEM and only the activations pass through shared memory; each CTA loads half of them.
//
// Persistent: pair p takes the tiles p, p + pairs, ... Per step of 128 inputs, numbered through over the pair's tiles:
//   warp 0      TMA: this CTA's half of the activations' tile (completion counted on the LEADER's barrier)
//   warp 2      TMA: the codes of its 128 weight rows, 128 bytes of a row (two steps) at a time
//   warps 12-27 four groups of four, steps in turn: unpack 128 codes of one weight row per thread into its TMEM lane
//   warp 1      leader only: tcgen05.mma.cta_group::2 kind::f16 with A in TMEM (M = 256, N = columns, K = 16) x 8
//   warps 4-11  the finished tile: TMEM -> registers -> y, 32 consecutive outputs of a row per store
// TMEM holds one accumulator (256 columns) and four unpacked steps (4 x 64). A tile's MMAs wait for the accumulator of the
// tile before to be read; the loads and the unpacking of up to four steps run ahead meanwhile.
#pragma once
#include "ptx.cuh"
#include "w4a16_gemm.cuh"
#include "w4a16_swap_gemm.cuh"

namespace qi {
namespace w4a16_pair_swap {

using w4a16_swap::load_scale_pair;
using w4a16_swap::unpack_step;

constexpr int BK = 128, BN = 128;         // inputs per step; weight rows per CTA
constexpr int MAX_COLUMNS = 256;          // activation rows of a tile; each CTA loads half of them
constexpr int PRODUCER_WARP = 0, MMA_WARP = 1, CODE_WARP = 2, EPILOGUE_WARP0 = 4, EPILOGUE_WARPS = 8, UNPACK_WARP0 = 12;
constexpr int UNPACK_GROUPS = 4, UNPACK_WARPS = 4 * UNPACK_GROUPS;
constexpr int THREADS = 32 * (UNPACK_WARP0 + UNPACK_WARPS);
constexpr int A_SLOTS = 4, A_COLUMNS = BK / 2, TMEM_COLUMNS = 512;
static_assert(MAX_COLUMNS + A_SLOTS * A_COLUMNS <= TMEM_COLUMNS && A_SLOTS == UNPACK_GROUPS, "accumulator and unpacked steps");
constexpr int STAGES = 5, HALF_BYTES = MAX_COLUMNS / 2 * 128, X_BYTES = 2 * HALF_BYTES;  // a stage: two boxes of 64 inputs
constexpr int CODE_STAGES = 4, CODE_BYTES = BN * 128, CODE_READERS = 8;                  // a chunk of codes: two steps, two groups read it
static_assert(CODE_STAGES == 2 || CODE_STAGES >= 4, "a group reads every second chunk: see w4a16_swap::smem_plan");
static_assert(STAGES >= A_SLOTS, "a stage's release stands for that of the slot of the step four before");
constexpr int BARRIER_BYTES = 256;
constexpr int SMEM_BYTES = STAGES * X_BYTES + CODE_STAGES * CODE_BYTES + BARRIER_BYTES + 1024;
static_assert(SMEM_BYTES <= 232448 && SMEM_BYTES >= ONE_CTA_SMEM, "one CTA per SM: see grid_release()");
static_assert((2 * STAGES + 2 * CODE_STAGES + A_SLOTS + 2) * 8 + 4 <= BARRIER_BYTES, "barrier block");
constexpr uint32_t AHEAD_BACKOFF_NS = 100, UNPACK_BACKOFF_NS = 20;

__device__ __forceinline__ void umma_f16_pair_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The wait for a copy out of TMEM, with its registers tied to it.
__device__ __forceinline__ void tmem_wait_16(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

// The order of the tiles: blocks of group_m rows of tiles; within a block the rows come first. The unpack warps, which run
// ahead, ask past the last tile too: there is no row of tiles left to divide by then, and the place is beyond the matrix.
struct TilePlace {
    int m_index, n_index;
};
__host__ __device__ constexpr TilePlace tile_place(int tile, int tiles_m, int tiles_n, int group_m) {
    if (tile >= tiles_m * tiles_n) return {0, tiles_n};
    const int of_block = group_m * tiles_n, block = tile / of_block, first = block * group_m;
    const int within = tile - block * of_block, rows = tiles_m - first < group_m ? tiles_m - first : group_m;
    return {first + within % rows, within / rows};
}
// Every tile once, nothing inside the matrix past the last; a division by zero would not compile.
constexpr bool covers(int tiles_m, int tiles_n, int group_m, int past) {
    bool seen[64] = {};
    for (int tile = 0; tile < tiles_m * tiles_n + past; ++tile) {
        const TilePlace at = tile_place(tile, tiles_m, tiles_n, group_m);
        if (tile >= tiles_m * tiles_n) {
            if (at.n_index < tiles_n) return false;
            continue;
        }
        if (at.m_index < 0 || at.m_index >= tiles_m || at.n_index < 0 || at.n_index >= tiles_n || seen[at.m_index * tiles_n + at.n_index]) return false;
        seen[at.m_index * tiles_n + at.n_index] = true;
    }
    return true;
}
static_assert(covers(1, 1, 1, 300) && covers(7, 5, 7, 80) && covers(8, 8, 8, 80) && covers(13, 4, 8, 80) && covers(17, 3, 8, 80) && covers(16, 4, 8, 80), "the walk over the tiles");

// `columns`: activation rows of a tile, a multiple of 16. PAIRED: see load_scale_pair.
template <bool PAIRED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_codes,
            const __half *__restrict__ scales, const __half *__restrict__ minimums,
            const float *__restrict__ bias, void *__restrict__ y, const GemmShape shape, const int columns, const int group_m) {
    extern __shared__ uint8_t smem_raw[];
    // the same offsets in both CTAs: the dynamic shared window starts at the same address in each
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smem_c = smem + STAGES * X_BYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_c + CODE_STAGES * CODE_BYTES);  // the leader's: both CTAs' activations
    uint64_t *empty = full + STAGES;
    uint64_t *code_full = empty + STAGES;
    uint64_t *code_empty = code_full + CODE_STAGES;
    uint64_t *a_ready = code_empty + CODE_STAGES;   // the leader's: both CTAs' unpack warps
    uint64_t *tile_full = a_ready + A_SLOTS;
    uint64_t *tile_empty = tile_full + 1;           // the leader's: both CTAs' epilogue warps
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tile_empty + 1);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int cta = static_cast<int>(cluster_ctarank());  // 0 = leader
    const int pair = static_cast<int>(blockIdx.x >> 1), pairs = static_cast<int>(gridDim.x >> 1);
    const int tiles_m = (shape.m + columns - 1) / columns, tiles_n = (shape.n + 2 * BN - 1) / (2 * BN), tiles = tiles_m * tiles_n;
    auto place = [&](int tile, int &m_index, int &n_index) {
        const TilePlace at = tile_place(tile, tiles_m, tiles_n, group_m);
        m_index = at.m_index, n_index = at.n_index;
    };
    // An even number of steps, as a chunk of codes holds two; one past the end loads, unpacks and multiplies nothing, it only
    // passes the barriers (320 inputs are 3 of 4 steps: 3000 x 18432 79.9 -> 74.7 us; 3000 x 3072 x 1088 35.3 -> 31.8).
    const int groups = shape.k / 64, steps = (groups + 3) / 4 * 2, real_steps = (groups + 1) / 2;
    const int half_bytes = columns / 2 * 128;                       // 64 inputs of this CTA's activation rows

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbarrier_init(&full[s], 1);
            mbarrier_init(&empty[s], 1);
        }
        for (int s = 0; s < CODE_STAGES; ++s) {
            mbarrier_init(&code_full[s], 1);
            mbarrier_init(&code_empty[s], CODE_READERS);
        }
        for (int s = 0; s < A_SLOTS; ++s) mbarrier_init(&a_ready[s], 2 * 4);
        mbarrier_init(tile_full, 1);
        mbarrier_init(tile_empty, 2 * EPILOGUE_WARPS);
        fence_barrier_init();
    }
    if (warp == MMA_WARP) {
        tmem_alloc_pair(tmem_slot, TMEM_COLUMNS);
        tmem_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before anything arrives on them from the other side
    tcgen05_fence_after();
    grid_wait();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + MAX_COLUMNS;
    const uint32_t full_u = smem_u32(full), empty_u = smem_u32(empty), code_full_u = smem_u32(code_full), code_empty_u = smem_u32(code_empty);
    const uint32_t a_ready_u = smem_u32(a_ready), tile_full_u = smem_u32(tile_full), tile_empty_u = smem_u32(tile_empty);
    bool alive = true;

    // The single-threaded roles run as converged warps with one elected lane (see w4a16_swap_gemm.cuh).
    if (warp == PRODUCER_WARP) {
        if (elect_one()) prefetch_tensormap(&map_x);
        const uint32_t x_u = smem_u32(smem);
        uint32_t s = 0, phase = 1;
        for (int tile = pair; tile < tiles && alive; tile += pairs) {
            int m_index, n_index;
            place(tile, m_index, n_index);
            const int m0 = m_index * columns + cta * (columns / 2);
            for (int step = 0; step < steps; ++step) {
                if (!mbarrier_wait_uniform(empty_u + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0xA000 | s, AHEAD_BACKOFF_NS)) { alive = false; break; }
                if (step >= real_steps) {
                    if (cta == 0 && elect_one()) mbarrier_arrive_u32(full_u + s * 8);
                } else if (elect_one()) {
                    if (cta == 0) mbarrier_arrive_expect_tx_u32(full_u + s * 8, 4 * half_bytes);  // both CTAs' boxes
                    tma_load_2d_pair_u32(x_u + s * X_BYTES, &map_x, full_u + s * 8, step * BK, m0);
                    tma_load_2d_pair_u32(x_u + s * X_BYTES + HALF_BYTES, &map_x, full_u + s * 8, step * BK + 64, m0);
                }
                __syncwarp();
                if (++s == STAGES) s = 0, phase ^= 1;
            }
        }
    } else if (warp == CODE_WARP) {
        if (elect_one()) prefetch_tensormap(&map_codes);
        const uint32_t c_u = smem_u32(smem_c);
        uint32_t s = 0, phase = 1;
        for (int tile = pair; tile < tiles && alive; tile += pairs) {
            int m_index, n_index;
            place(tile, m_index, n_index);
            const int n0 = n_index * (2 * BN) + cta * BN;
            for (int step = 0; step < steps; step += 2) {
                if (!mbarrier_wait_uniform(code_empty_u + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0xA200 | s, AHEAD_BACKOFF_NS)) { alive = false; break; }
                if (elect_one()) {
                    mbarrier_arrive_expect_tx_u32(code_full_u + s * 8, CODE_BYTES);
                    tma_load_2d_u32(c_u + s * CODE_BYTES, &map_codes, code_full_u + s * 8, step * (BK / 2), n0);
                }
                __syncwarp();
                if (++s == CODE_STAGES) s = 0, phase ^= 1;
            }
        }
    } else if (warp == MMA_WARP) {
        if (cta == 0) {
            const uint32_t idesc = umma_idesc_f16_f32(2 * BN, 0) | (static_cast<uint32_t>(columns >> 3) << 17);
            const uint64_t b_first = umma_desc_k_sw128(smem_u32(smem));
            uint32_t s = 0, phase = 0, slot = 0, slot_phase = 0, tile_phase = 1;
            for (int tile = pair; tile < tiles && alive; tile += pairs, tile_phase ^= 1) {
                if (!mbarrier_wait_uniform(tile_empty_u, tile_phase, &g_status, STATUS_WAIT_TMEM_EMPTY | 0xA000)) break;
                for (int step = 0; step < steps; ++step) {
                    if (!mbarrier_wait_uniform2(full_u + s * 8, phase, a_ready_u + slot * 8, slot_phase, &g_status, STATUS_WAIT_READY | 0xA000 | s)) { alive = false; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint64_t b_desc = b_first + s * (X_BYTES >> 4);
                        const uint32_t a = tmem_a + slot * A_COLUMNS;
                        if (step < real_steps) {
#pragma unroll
                            for (int kk = 0; kk < BK / 16; ++kk)
                                umma_f16_pair_a_tmem(tmem_base, a + kk * 8, b_desc + (kk >> 2) * (HALF_BYTES >> 4) + (kk & 3) * 2, idesc, (step | kk) != 0 ? 1u : 0u);
                        }
                        tcgen05_commit_pair(&empty[s]);
                        if (step + 1 == steps) tcgen05_commit_pair(tile_full);
                    }
                    __syncwarp();
                    if (++s == STAGES) s = 0, phase ^= 1;
                    if (++slot == A_SLOTS) slot = 0, slot_phase ^= 1;
                }
            }
        }
    } else if (warp >= UNPACK_WARP0) {
        const int quadrant = warp & 3, group = (warp - UNPACK_WARP0) >> 2;
        const int local_row = quadrant * 32 + lane;
        const uint32_t tmem_lane = tmem_a + group * A_COLUMNS + (static_cast<uint32_t>(quadrant * 32) << 16);
        const uint32_t leader_ready = map_to_cta(a_ready_u + group * 8, 0);
        // Step `group`, then every fourth, over all tiles. The chunk of codes: two steps each, so two chunks on every time.
        int tile = pair, step = group;
        while (step >= steps) step -= steps, tile += pairs;
        uint32_t chunk = group / 2, chunk_phase = 0;
        int before = group - A_SLOTS, before_phase = 0;  // the stage of the step four before, whose release frees the slot
        const __half *row_scales = scales, *row_minimums = minimums;
        bool inside = false;
        auto at_tile = [&]() {
            int m_index, n_index;
            place(tile, m_index, n_index);
            const int row = n_index * (2 * BN) + cta * BN + local_row;
            inside = row < shape.n;  // past the last tile no row is
            row_scales = scales + static_cast<size_t>(inside ? row : 0) * groups;
            row_minimums = minimums + static_cast<size_t>(inside ? row : 0) * groups;
        };
        at_tile();
        uint32_t scale_next = load_scale_pair<PAIRED>(row_scales, 2 * step, groups, inside);
        uint32_t minimum_next = load_scale_pair<PAIRED>(row_minimums, 2 * step, groups, inside);
#pragma unroll 1
        while (tile < tiles) {
            const uint32_t scale = scale_next, minimum = minimum_next;
            const int piece = (step & 1) * 4;
            const bool real = step < real_steps;
            step += UNPACK_GROUPS;
            if (step >= steps) {
                while (step >= steps) step -= steps, tile += pairs;
                at_tile();
            }
            scale_next = load_scale_pair<PAIRED>(row_scales, 2 * step, groups, inside);
            minimum_next = load_scale_pair<PAIRED>(row_minimums, 2 * step, groups, inside);
            if (!mbarrier_wait_uniform(code_full_u + chunk * 8, chunk_phase, &g_status, STATUS_WAIT_FULL | 0xA100 | chunk, UNPACK_BACKOFF_NS)) break;
            const auto slot_free = [&]() {  // without it a step past the end could say that it is ready before the one it follows was read
                if (before >= 0 && !mbarrier_wait_uniform(empty_u + before * 8, before_phase, &g_status, STATUS_WAIT_EMPTY | 0xA100 | group, UNPACK_BACKOFF_NS)) alive = false;
                tcgen05_fence_after();
            };
            if (real) unpack_step(smem_c + chunk * CODE_BYTES + local_row * 128, piece, local_row & 7, scale, minimum, tmem_lane, slot_free);
            else slot_free();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbarrier_arrive_cluster(leader_ready);
                mbarrier_arrive_u32(code_empty_u + chunk * 8);
            }
            if (!alive) break;
            chunk += UNPACK_GROUPS / 2;
            if (chunk >= CODE_STAGES) chunk -= CODE_STAGES, chunk_phase ^= 1;
            before += A_SLOTS;
            if (before >= STAGES) before -= STAGES, before_phase ^= 1;
        }
    } else if (warp >= EPILOGUE_WARP0) {
        // Two warps per TMEM quadrant, sixteen columns at a time in turn. The tensor cores wait meanwhile, so the next
        // sixteen are on their way while a warp converts and stores.
        const int quadrant = warp & 3, half = (warp - EPILOGUE_WARP0) >> 2;
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quadrant * 32) << 16), leader_tile_empty = map_to_cta(tile_empty_u, 0);
        uint32_t phase = 0;
        for (int tile = pair; tile < tiles; tile += pairs, phase ^= 1) {
            int m_index, n_index;
            place(tile, m_index, n_index);
            const int m0 = m_index * columns, n = n_index * (2 * BN) + cta * BN + quadrant * 32 + lane;
            const int rows = shape.m - m0 < columns ? shape.m - m0 : columns;
            const bool inside = n < shape.n;
            const float add = bias != nullptr && inside ? __ldg(bias + n) : 0.0f;
            if (!mbarrier_wait_uniform(tile_full_u, phase, &g_status, STATUS_WAIT_TMEM_FULL | 0xA000, AHEAD_BACKOFF_NS)) break;
            tcgen05_fence_after();
            uint32_t r[2][16];
            auto store = [&](const uint32_t (&v)[16], int c) {
                if (!inside) return;
                const size_t element = static_cast<size_t>(m0 + c) * shape.ldy + n;
                const int some = rows - c;
                if (shape.y_is_half) {
                    __half *out = static_cast<__half *>(y) + element;
#pragma unroll
                    for (int j = 0; j < 16; ++j, out += shape.ldy)
                        if (j < some) *out = __float2half_rn(__uint_as_float(v[j]) + add);
                } else {
                    float *out = static_cast<float *>(y) + element;
#pragma unroll
                    for (int j = 0; j < 16; ++j, out += shape.ldy)
                        if (j < some) *out = __uint_as_float(v[j]) + add;
                }
            };
            const int c0 = half * 16;
            if (c0 < columns) tmem_load_32x16(tmem_lane + c0, r[0]);
#pragma unroll 1
            for (int c = c0; c < columns; c += 64) {
                tmem_wait_16(r[0]);
                if (c + 32 < columns) tmem_load_32x16(tmem_lane + c + 32, r[1]);
                store(r[0], c);
                if (c + 32 >= columns) break;
                tmem_wait_16(r[1]);
                if (c + 64 < columns) tmem_load_32x16(tmem_lane + c + 64, r[0]);
                store(r[1], c + 32);
            }
            tmem_load_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbarrier_arrive_cluster(leader_tile_empty);
        }
    }

    // teardown: nothing of this CTA may still be in flight when TMEM and shared memory go away
    tcgen05_fence_before();
    __syncthreads();
    if (*reinterpret_cast<volatile uint32_t *>(&g_status) != 0) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);  // a wait gave up: let bulk copies that were already issued land
    }
    __syncwarp();
    cluster_sync();  // neither CTA may leave while the other can still reach its shared memory or barriers
    if (warp == MMA_WARP) {
        __syncwarp();
        tcgen05_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLUMNS);
    }
}

}  // namespace w4a16_pair_swap
}  // namespace qi

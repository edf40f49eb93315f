// W4A16 g64 GEMV for 1..8 activation rows, streaming form: same operator and arithmetic as w4a16_gemv.cuh
// (the reference's w4a16_gemm_kernel, qwen_image_cuda/cuda/gemm.cu:191-268, without its padding of the rows
// to 128), for matrices whose rows are short enough that 16 of them fit a shared-memory stage (K <= 4096).
//
// A CTA per SM walks over tiles of 16 weight rows. A tile's codes, scales and minimums are three contiguous ranges of the
// pack (16 whole rows each), so one thread fetches them with three bulk asynchronous copies (cp.async.bulk, completion
// counted on an mbarrier) into a ring of up to eight stages, and the copies of the next tiles are in flight while the
// warps unpack. The tiles in the ring are dealt out to four teams of six warps; within a tile the team's warps split K:
// lane (r, q) = (lane / 4, lane % 4) takes 32 codes (half a group) of rows r and r + 8 per step, unpacks them, and
// feeds them as the A operand of mma.sync.m16n8k16 (fp32 accumulate) whose B operand carries up to 8 activation rows;
// the order of k inside an MMA is free as long as both operands agree. The K slices are summed through shared memory in a
// fixed order. The teams have a barrier each and drift apart: against two CTAs of eight warps with two CTA-wide barriers
// per tile, 18432 x 3072 went from 14.7 to 11.9 us alone and from 9.1 to 7.5 us in groups of 60 (512 threads: 12.2 and
// 7.9; 1024: 11.6 and 8.0).
//
// Unpacking is what the SMs spend their time on (18432 x 3072 in groups of 60: the copies alone 4.6 us a matrix; before,
// 62 % of the integer pipe and 205 instructions per 2048 weights, 7.5 us; now 167 and 6.3 us; alone 11.9 -> 10.8), so it is
// cut to ten instructions per eight weights. A nibble moved to bits 2..5 or 6..9 of a 16-bit lane is the fp16 denormal
// code * 2^-22 or code * 2^-18, so one shift serves two nibbles; one half2 fused multiply-add with the scale times 2^22 or
// 2^18 and the minimum gives fp16(code * scale + minimum) with a single rounding, which is what the reference's
// __float2half(fmaf(code, scale, minimum)) gives whenever |w| <= 1 (gemm.cu:229-230; see w4a16_gemm.cuh). A word of eight
// nibbles yields the pairs (0,4), (1,5), (2,6), (3,7); the activations are stored once per CTA in shared memory in that
// order. A scale of 1/64 or more, whose 2^22-fold is no fp16 number, sends the warp's step down a path in which the smaller
// multiple alone is used (below 1/4), or down the slowest, with each code made an fp16 integer first.
#pragma once
#include "ptx.cuh"
#include "w4a16_gemv.cuh"

namespace qi {
namespace w4a16 {

constexpr int STREAM_THREADS = 768, STREAM_MAX_STAGES = 8, STREAM_ROWS = 16;
constexpr int STREAM_TEAMS = 4, STREAM_TEAM_WARPS = STREAM_THREADS / 32 / STREAM_TEAMS;
constexpr int STREAM_MAX_K = 4096;  // 16 rows of codes, scales and minimums: 36 KB per stage

__host__ __device__ constexpr int stream_stage_bytes(int k) { return STREAM_ROWS * (k / 2) + 2 * STREAM_ROWS * (k / 64) * 2; }
// a row of activations: a step's 16 pieces of 16 bytes, the four lanes' first pieces, their second, ...; 64 bytes more
// set the next row on the other banks
__host__ __device__ constexpr int stream_x_pieces(int k) { return (k + 127) / 128 * 16 + 4; }
__host__ __device__ constexpr int stream_x_bytes(int m, int k) { return m * stream_x_pieces(k) * 16; }

// global -> shared, any multiple of 16 bytes, both addresses 16-byte aligned; completion on an mbarrier of this CTA
__device__ __forceinline__ void bulk_load(void *smem, const void *global, uint32_t bytes, uint64_t *barrier) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem)),
                 "l"(global), "r"(bytes), "r"(smem_u32(barrier))
                 : "memory");
}

// Eight nibbles of one row -> four half2 of dequantised weights, pairs (0,4), (1,5), (2,6), (3,7). A nibble at bits 2..5 of
// a 16-bit lane is code * 2^-22 and takes the scale times 2^22, at bits 6..9 it is code * 2^-18 and takes it times 2^18.
// LARGE: the scale times 2^18 only, the nibbles at bits 2..5 times 16 first (exact).
template <bool LARGE>
__device__ __forceinline__ void unpack_word(uint32_t word, __half2 scale_22, __half2 scale_18, __half2 minimum2, uint32_t (&out)[4]) {
    const uint32_t up = word << 2, down = word >> 6;
    const uint32_t moved[4] = {up & 0x003C003Cu, up & 0x03C003C0u, down & 0x003C003Cu, down & 0x03C003C0u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        __half2 code = *reinterpret_cast<const __half2 *>(&moved[j]);
        if (LARGE && j % 2 == 0) code = __hmul2(code, scale_22);  // sixteen
        const __half2 weight = __hfma2(code, !LARGE && j % 2 == 0 ? scale_22 : scale_18, minimum2);
        out[j] = *reinterpret_cast<const uint32_t *>(&weight);
    }
}

// The same pairs for any scale: each code as an fp16 integer, then the same fused multiply-add.
__device__ __forceinline__ void unpack_word_any_scale(uint32_t word, __half2 scale2, __half2 minimum2, uint32_t (&out)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 code = __halves2half2(__ushort2half_rn(static_cast<unsigned short>((word >> (4 * j)) & 15u)),
                                            __ushort2half_rn(static_cast<unsigned short>((word >> (4 * j + 16)) & 15u)));
        const __half2 weight = __hfma2(code, scale2, minimum2);
        out[j] = *reinterpret_cast<const uint32_t *>(&weight);
    }
}

// Several matrices of one shape for one launch: the grouped form walks the tiles of all of them as one list, so
// that the launch, the first copies and the staging of the activations are paid once. The table travels in the
// kernel's parameters (40 bytes per matrix).
constexpr int STREAM_GROUP = 64;
struct StreamItem {
    const uint8_t *codes;
    const __half *scales, *minimums;
    const float *bias;
    void *y;
};
struct StreamItems {
    StreamItem item[STREAM_GROUP];
};

// Dynamic shared memory: `stages` stages of stream_stage_bytes(k), then the activations (stream_x_bytes(m, k)).
// GROUPED: `count` matrices [n, k] from `group`, tile t of the launch is tile t % (n / 16) of matrix t / (n / 16);
// otherwise the one matrix given by the pointer arguments.
template <bool GROUPED>
__device__ __forceinline__ void gemv_stream_body(const __half *__restrict__ x, const uint8_t *__restrict__ codes, const __half *__restrict__ scales,
                   const __half *__restrict__ minimums, const float *__restrict__ bias, void *__restrict__ y,
                   int m, int n, int k, long long ldy, int y_is_half, int stages, const StreamItems *group, int count) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    __shared__ uint64_t full[STREAM_MAX_STAGES];
    __shared__ volatile int fetched[STREAM_MAX_STAGES];  // the tile that was last sent for into each stage
    __shared__ alignas(8) float partials[STREAM_TEAMS][2][STREAM_TEAM_WARPS][16][8];
    const int team = threadIdx.x / (STREAM_TEAM_WARPS * 32), warp = threadIdx.x / 32 % STREAM_TEAM_WARPS, lane = threadIdx.x & 31;
    const int team_thread = threadIdx.x % (STREAM_TEAM_WARPS * 32);
    const int r = lane >> 2, q = lane & 3;
    const int groups = k / 64, steps = (groups + 1) / 2;  // a step: two groups, a quarter of the lanes on each half group
    const int code_bytes = STREAM_ROWS * (k / 2), scale_bytes = STREAM_ROWS * groups * 2;
    const int stage_bytes = code_bytes + 2 * scale_bytes;
    const int tiles_each = n / STREAM_ROWS, tiles = GROUPED ? tiles_each * count : tiles_each;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbarrier_init(&full[s], 1);
            fetched[s] = -1;
        }
        fence_barrier_init();
    }
    grid_wait();
    grid_release();
    // the activations, once per CTA, every eight inputs in the order (0,4,1,5,2,6,3,7) the unpacked pairs have
    uint4 *x_pairs = reinterpret_cast<uint4 *>(smem + static_cast<size_t>(stages) * stage_bytes);
    const int x_row = stream_x_pieces(k);
    for (int item = threadIdx.x; item < m * steps * 16; item += STREAM_THREADS) {
        const int row = item / (steps * 16), piece = item % (steps * 16);  // input / 8; a ragged last step is filled with zeros
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (piece < k / 8) v = __ldg(reinterpret_cast<const uint4 *>(x) + static_cast<size_t>(row) * (k / 8) + piece);
        x_pairs[row * x_row + piece / 16 * 16 + piece % 4 * 4 + piece / 4 % 4] =
            make_uint4(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.x, v.z, 0x7632), __byte_perm(v.y, v.w, 0x5410), __byte_perm(v.y, v.w, 0x7632));
    }
    __syncthreads();
    auto fetch = [&](int tile, int s) {  // one thread
        uint8_t *stage = smem + static_cast<size_t>(s) * stage_bytes;
        const int of_launch = tile;
        const uint8_t *from_codes = codes;
        const __half *from_scales = scales, *from_minimums = minimums;
        if (GROUPED) {
            const StreamItem &item = group->item[tile / tiles_each];
            from_codes = item.codes, from_scales = item.scales, from_minimums = item.minimums;
            tile %= tiles_each;
        }
        const size_t row0 = static_cast<size_t>(tile) * STREAM_ROWS;
        mbarrier_arrive_expect_tx(&full[s], static_cast<uint32_t>(stage_bytes));
        bulk_load(stage, from_codes + row0 * (k / 2), code_bytes, &full[s]);
        bulk_load(stage + code_bytes, from_scales + row0 * groups, scale_bytes, &full[s]);
        bulk_load(stage + code_bytes + scale_bytes, from_minimums + row0 * groups, scale_bytes, &full[s]);
        __threadfence_block();
        fetched[s] = of_launch;
    };
    if (threadIdx.x == 0) {
        int tile = blockIdx.x;
        for (int s = 0; s < stages && tile < tiles; ++s, tile += gridDim.x) fetch(tile, s);
    }

    const __half nothing = __ushort_as_half(0);
    const __half2 sixty_fourth = __float2half2_rn(1.0f / 64.0f), quarter = __float2half2_rn(0.25f), two_to_9 = __float2half2_rn(512.0f), sixteen = __float2half2_rn(16.0f);
    // Activation row lane / 4 is the B operand's column of that number, and a column only ever meets its own results: a
    // lane past the last row feeds row 0 again, and what comes of it is not stored.
    const uint4 *my_x = x_pairs + (r < m ? r : 0) * x_row + q;
    // Team t takes the CTA's tiles t, t + 4, ...; tile i of the CTA lies in stage i modulo the number of stages.
    uint32_t s = team, phase = 0;
    while (s >= static_cast<uint32_t>(stages)) s -= stages, phase ^= 1;
    int parity = 0;
    bool gave_up = false;
    for (int tile = blockIdx.x + team * gridDim.x; tile < tiles; tile += STREAM_TEAMS * gridDim.x, parity ^= 1) {
        float (&partial)[STREAM_TEAM_WARPS][16][8] = partials[team][parity];
        // The stage's last user may have been another team. Only once this tile has been sent for is the phase before complete,
        // and the parity of this one's unambiguous.
        const bool arrived = wait_uniform([&]() { return fetched[s] == tile; }, &g_status, STATUS_WAIT_EMPTY | 0xB000 | s, 32) &&
                             mbarrier_wait_uniform(smem_u32(&full[s]), phase, &g_status, STATUS_WAIT_FULL | 0xB000 | s);
        const uint8_t *stage = smem + static_cast<size_t>(s) * stage_bytes;
        const __half *stage_scales = reinterpret_cast<const __half *>(stage + code_bytes);
        const __half *stage_minimums = reinterpret_cast<const __half *>(stage + code_bytes + scale_bytes);
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (arrived) {
            for (int step = warp; step < steps; step += STREAM_TEAM_WARPS) {
                const int g = 2 * step + (q >> 1);  // this lane's group; q & 1 is the half of it
                const uint8_t *my_codes = stage + r * (k / 2) + step * 64 + q * 16;
                const uint4 code_a = *reinterpret_cast<const uint4 *>(my_codes);
                const uint4 code_b = *reinterpret_cast<const uint4 *>(my_codes + 8 * (k / 2));
                __half scale_a = stage_scales[r * groups + g], scale_b = stage_scales[(r + 8) * groups + g];
                __half minimum_a = stage_minimums[r * groups + g], minimum_b = stage_minimums[(r + 8) * groups + g];
                if (2 * step + 1 >= groups && q >= 2) {  // past a ragged end: what was read lies in the CTA's shared memory; zeros
                    scale_a = scale_b = minimum_a = minimum_b = nothing;
                }
                const uint32_t wa[4] = {code_a.x, code_a.y, code_a.z, code_a.w};
                const uint32_t wb[4] = {code_b.x, code_b.y, code_b.z, code_b.w};
                const __half2 ma = __half2half2(minimum_a), mb = __half2half2(minimum_b);
                const uint4 *px = my_x + step * 16;
                auto multiply = [&](auto unpack) {
#pragma unroll
                    for (int w = 0; w < 4; ++w) {  // 8 inputs of each row per word, two MMA steps
                        const uint4 xv = px[4 * w];
                        uint32_t pa[4], pb[4];
                        unpack(wa[w], wb[w], pa, pb);
                        const uint32_t first[4] = {pa[0], pb[0], pa[1], pb[1]}, second[4] = {pa[2], pb[2], pa[3], pb[3]};
                        mma_m16n8k16(c, first, xv.x, xv.y);
                        mma_m16n8k16(c, second, xv.z, xv.w);
                    }
                };
                // scale * 2^22 is an fp16 number below 1/64, scale * 2^18 below 1/4 (a NaN fails both tests)
                const __half2 magnitudes = __habs2(__halves2half2(scale_a, scale_b));
                if (__all_sync(0xffffffffu, __hblt2(magnitudes, sixty_fourth))) {
                    const __half2 sa = __hmul2(__hmul2(__half2half2(scale_a), two_to_9), two_to_9), sa_22 = __hmul2(sa, sixteen);
                    const __half2 sb = __hmul2(__hmul2(__half2half2(scale_b), two_to_9), two_to_9), sb_22 = __hmul2(sb, sixteen);
                    multiply([&](uint32_t a, uint32_t b, uint32_t(&pa)[4], uint32_t(&pb)[4]) {
                        unpack_word<false>(a, sa_22, sa, ma, pa);
                        unpack_word<false>(b, sb_22, sb, mb, pb);
                    });
                } else if (__all_sync(0xffffffffu, __hblt2(magnitudes, quarter))) {
                    const __half2 sa = __hmul2(__hmul2(__half2half2(scale_a), two_to_9), two_to_9);
                    const __half2 sb = __hmul2(__hmul2(__half2half2(scale_b), two_to_9), two_to_9);
                    multiply([&](uint32_t a, uint32_t b, uint32_t(&pa)[4], uint32_t(&pb)[4]) {
                        unpack_word<true>(a, sixteen, sa, ma, pa);
                        unpack_word<true>(b, sixteen, sb, mb, pb);
                    });
                } else {
                    const __half2 sa = __half2half2(scale_a), sb = __half2half2(scale_b);
                    multiply([&](uint32_t a, uint32_t b, uint32_t(&pa)[4], uint32_t(&pb)[4]) {
                        unpack_word_any_scale(a, sa, ma, pa);
                        unpack_word_any_scale(b, sb, mb, pb);
                    });
                }
            }
        }
        // c[0], c[1]: weight row r, activation rows 2q, 2q+1; c[2], c[3]: weight row r + 8
        *reinterpret_cast<float2 *>(&partial[warp][r][2 * q]) = make_float2(c[0], c[1]);
        *reinterpret_cast<float2 *>(&partial[warp][r + 8][2 * q]) = make_float2(c[2], c[3]);
        // The team is done with the stage, and the partial sums are complete. The sums alternate between two places: those of
        // this tile are read below and written again two tiles on, with the next tile's barrier in between.
        named_barrier_sync(1 + team, STREAM_TEAM_WARPS * 32);
        gave_up |= !arrived;
        if (team_thread == 0 && arrived) {
            const int next = tile + stages * gridDim.x;
            if (next < tiles) fetch(next, s);
        }
        // fixed-order sum over the K slices: thread -> (activation row, weight row), so that few rows keep few warps
        const int b = team_thread >> 4, row = team_thread & 15;
        if (b < m) {
            const float *to_bias = bias;
            void *to_y = y;
            int local_tile = tile;
            if (GROUPED) {
                const StreamItem &item = group->item[tile / tiles_each];
                to_bias = item.bias, to_y = item.y;
                local_tile = tile % tiles_each;
            }
            const int out_row = local_tile * STREAM_ROWS + row;
            float total = 0.0f;
#pragma unroll
            for (int slice = 0; slice < STREAM_TEAM_WARPS; ++slice) total += partial[slice][row][b];
            if (to_bias != nullptr) total += __ldg(to_bias + out_row);
            if (y_is_half) static_cast<__half *>(to_y)[static_cast<size_t>(b) * ldy + out_row] = __float2half_rn(total);
            else static_cast<float *>(to_y)[static_cast<size_t>(b) * ldy + out_row] = total;
        }
        s += STREAM_TEAMS;
        while (s >= static_cast<uint32_t>(stages)) s -= stages, phase ^= 1;
    }
    // Every copy has a team that waits for it. Where a wait gave up, let the copies already issued land. (Asking the status
    // word instead is a round trip to L2 at the end of every CTA: 4080 x 4096 5.6 -> 5.9 us.)
    if (gave_up) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
}

__global__ void __launch_bounds__(STREAM_THREADS, 1)
gemv_stream_kernel(const __half *__restrict__ x, const uint8_t *__restrict__ codes, const __half *__restrict__ scales,
                   const __half *__restrict__ minimums, const float *__restrict__ bias, void *__restrict__ y,
                   int m, int n, int k, long long ldy, int y_is_half, int stages) {
    gemv_stream_body<false>(x, codes, scales, minimums, bias, y, m, n, k, ldy, y_is_half, stages, nullptr, 1);
}

__global__ void __launch_bounds__(STREAM_THREADS, 1)
gemv_stream_grouped_kernel(const __half *__restrict__ x, const __grid_constant__ StreamItems group, int count,
                           int m, int n, int k, long long ldy, int y_is_half, int stages) {
    gemv_stream_body<true>(x, nullptr, nullptr, nullptr, nullptr, nullptr, m, n, k, ldy, y_is_half, stages, &group, count);
}

}  // namespace w4a16
}  // namespace qi

// W4A16 g64 GEMV for 1..8 activation rows, streaming form: same operator and arithmetic as w4a16_gemv.cuh
// (the reference's w4a16_gemm_kernel, qwen_image_cuda/cuda/gemm.cu:191-268, without its padding of the rows
// to 128), for matrices whose rows are short enough that 16 of them fit a shared-memory stage (K <= 4096).
//
// A CTA per SM walks over tiles of 16 weight rows. A tile's codes, scales and minimums are three contiguous ranges of the
// pack (16 whole rows each), so one thread, in a warp of its own, fetches them with three or four bulk asynchronous copies
// (cp.async.bulk, completion counted on an mbarrier) into a ring of up to sixteen stages, and the copies of the next tiles
// are in flight while the others unpack. The tiles in the ring are dealt out to teams of warps; within a tile the team's
// warps split K: lane (r, q) = (lane / 4, lane % 4) takes the 64 codes of one group of two weight rows per step, unpacks
// them, and feeds them as rows r and r + 8 of the A operand of mma.sync.m16n8k16 (fp32 accumulate) whose B operand carries up
// to 8 activation rows; the order of k inside an MMA is free as long as both operands agree. K is cut into slices, by k alone,
// and in each the first and the second halves of the groups are added up apart: an MMA cuts its sum to 24 bits, always towards
// zero, so that the error grows with the number of MMAs in a chain (18432 x 3072 against 64 bits, 2-norm: 1.25e-6 with
// chains of 64, 6.4e-7 with chains of 32). The sums of the halves, then of the slices, are added through shared memory in a
// fixed order. A team has a warp for each slice, which keeps both halves' sums, or (HALVES) two, a half each: a tile is done sooner
// but takes more instructions, and the bits are the same. So a row of activations alone, among others, against a slice of a
// matrix, a whole one or one in a group gives the same bits.
//
// What bounds it, 18432 x 3072 on cold weights: alone the first load, the copies (31.9 MB, 4.7 us) and the last tiles' steps;
// in groups of 60 instructions and copies about alike (5.0 us a matrix; the copies alone 4.6).
// What counted, in that order: shared memory by 32-bit addresses instead of generic pointers (76.0 -> 61.2 million
// warp instructions for sixteen matrices); a step of whole groups, which halves what a step spends on its scales; a warp
// that does nothing but fetch, since a thread that unpacks held its team up while the copy engine took its requests; and
// codes read without bank conflicts. Rows lie a multiple of 32 bytes apart, most often of 128, so the eight lanes that a
// 16-byte load serves at a time, four of each of two MMA rows, would meet on four banks. So the lower eight weight rows lie
// 16 bytes further on in the stage, by a copy of their own, and MMA rows of either parity are weight rows of either half. From
// K = 2048 on; below, the fourth copy of a tile costs more than the conflicts (18432 x 512 4.45 us without, 4.75 with it;
// 60 x 9216 x 1024 88 and 92; 18432 x 2048 7.4 without, 7.1 with it, 3072 x 2048 4.25 and 4.17).
// Before, odd weight rows read the two halves of their group in the other order, against columns of B that held the activations
// so. That order of sums is not there for more than four activation rows, whose bits differed from those of one row; it was
// also slower (m = 8: 18432 x 3072 11.4 -> 11.1 us, 12288 x 4096 13.4 -> 12.7).
// Measured without gain: two steps unrolled, a limit on the copies in flight, a warp that does nothing but the final sums
// (10.2 us alone), teams of 8 and 12 warps (10.7, 10.5), lanes that send for one range each (60 x 18432 x 512 150 us -> 217),
// two slices a warp one after the other, so that teams of three and of six had the same slices (60 x 18432 x 3072 300 ->
// 334), a second MMA for the rows past the fourth (8 x 18432 x 3072 11.3 -> 13.1).
//
// Unpacking takes ten instructions per eight weights. A nibble moved to bits 2..5 or 6..9 of a 16-bit lane is the fp16 denormal
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

// 24 warps unpack, one fetches
constexpr int STREAM_WARPS = 24, STREAM_THREADS = (STREAM_WARPS + 1) * 32, STREAM_MAX_STAGES = 16, STREAM_ROWS = 16;
constexpr uint32_t STREAM_MAX_SLICES = 6;
constexpr int STREAM_STEP_GROUPS = 4;  // a step of a warp: a group for each of a row's four lanes
constexpr int STREAM_MAX_K = 4096;  // 16 rows of codes, scales and minimums: 36 KB per stage
constexpr int STREAM_SHIFT_FROM = 2048;  // see above
// Bytes that the lower eight rows' codes lie further on in a stage.
__host__ __device__ constexpr int stream_shift(int k) { return k >= STREAM_SHIFT_FROM ? 16 : 0; }

__host__ __device__ constexpr int stream_stage_bytes(int k) { return STREAM_ROWS * (k / 2) + stream_shift(k) + 2 * STREAM_ROWS * (k / 64) * 2; }
// a row of activations in pieces of 16 bytes; 64 bytes more set the next row on the other banks
__host__ __device__ constexpr int stream_steps(int k) { return (k / 64 + STREAM_STEP_GROUPS - 1) / STREAM_STEP_GROUPS; }
__host__ __device__ constexpr int stream_x_pieces(int k) { return stream_steps(k) * STREAM_STEP_GROUPS * 8 + 4; }
__host__ __device__ constexpr int stream_x_bytes(int m, int k) { return m * stream_x_pieces(k) * 16; }
__host__ __device__ constexpr int stream_partial_bytes(int m) { return 2 * STREAM_WARPS * m * STREAM_ROWS * 4; }  // a warp's, twice
__host__ __device__ constexpr int stream_fixed_bytes(int m, int k) { return stream_x_bytes(m, k) + stream_partial_bytes(m) + 128; }

__device__ __forceinline__ uint4 lds_16(uint32_t address) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(address));
    return v;
}
__device__ __forceinline__ __half lds_half(uint32_t address) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(address));
    return __ushort_as_half(v);
}
__device__ __forceinline__ float lds_float(uint32_t address) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(address));
    return v;
}
__device__ __forceinline__ void sts_float(uint32_t address, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(address), "f"(v) : "memory"); }
__device__ __forceinline__ void sts_16(uint32_t address, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// global -> shared, any multiple of 16 bytes, both addresses 16-byte aligned; completion on an mbarrier of this CTA
__device__ __forceinline__ void bulk_load(uint32_t smem, const void *global, uint32_t bytes, uint32_t barrier) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem), "l"(global), "r"(bytes), "r"(barrier)
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

// Dynamic shared memory: `stages` stages of stream_stage_bytes(k), then the activations (stream_x_bytes(m, k)), then the
// teams' partial sums (stream_partial_bytes(m)).
// GROUPED: `count` matrices [n, k] from `group`, tile t of the launch is tile t % (n / 16) of matrix t / (n / 16);
// otherwise the one matrix given by the pointer arguments.
template <bool GROUPED, bool HALVES>
__device__ __forceinline__ void gemv_stream_body(const __half *__restrict__ x, const uint8_t *__restrict__ codes, const __half *__restrict__ scales,
                   const __half *__restrict__ minimums, const float *__restrict__ bias, void *__restrict__ y,
                   int m, int n, int k, long long ldy, int y_is_half, int stages, int team_warps, const StreamItems *group, int count) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem = (smem_u32(smem_raw) + 127) & ~127u;
    __shared__ uint64_t full[STREAM_MAX_STAGES], empty[STREAM_MAX_STAGES];
    __shared__ volatile int fetched[STREAM_MAX_STAGES];  // the tile that was last sent for into each stage
    const uint32_t full_u = smem_u32(full), empty_u = smem_u32(empty);
    const int cta_warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int teams = STREAM_WARPS / team_warps, team = cta_warp / team_warps, warp = cta_warp - team * team_warps;
    const int team_threads = team_warps * 32, team_thread = warp * 32 + lane;
    const uint32_t r = lane >> 2, q = lane & 3;
    const uint32_t groups = k / 64, steps = stream_steps(k), row_bytes = k / 2;
    const uint32_t code_bytes = STREAM_ROWS * row_bytes, scale_bytes = STREAM_ROWS * groups * 2;
    const uint32_t shift = stream_shift(k), scales_at = code_bytes + shift, stage_bytes = scales_at + 2 * scale_bytes;
    const int tiles_each = n / STREAM_ROWS, tiles = GROUPED ? tiles_each * count : tiles_each;
    const int step_tiles = static_cast<int>(gridDim.x);

    // one thread sends for a tile: its place among all and, GROUPED, its matrix and its place in that
    auto fetch = [&](int tile, int item_index, int local, uint32_t s) {
        const uint32_t stage = smem + s * stage_bytes, barrier = full_u + s * 8;
        const uint8_t *from_codes = codes;
        const __half *from_scales = scales, *from_minimums = minimums;
        if (GROUPED) {
            const StreamItem &item = group->item[item_index];
            from_codes = item.codes, from_scales = item.scales, from_minimums = item.minimums;
        }
        from_codes += static_cast<size_t>(local) * code_bytes;
        mbarrier_arrive_expect_tx_u32(barrier, code_bytes + 2 * scale_bytes);
        const uint32_t upper = shift != 0 ? code_bytes / 2 : code_bytes;
        bulk_load(stage, from_codes, upper, barrier);
        if (shift != 0) bulk_load(stage + upper + shift, from_codes + upper, upper, barrier);
        bulk_load(stage + scales_at, reinterpret_cast<const uint8_t *>(from_scales) + static_cast<size_t>(local) * scale_bytes, scale_bytes, barrier);
        bulk_load(stage + scales_at + scale_bytes, reinterpret_cast<const uint8_t *>(from_minimums) + static_cast<size_t>(local) * scale_bytes, scale_bytes, barrier);
        __threadfence_block();
        fetched[s] = tile;
    };
    if (threadIdx.x < stages) {
        mbarrier_init(&full[threadIdx.x], 1);
        mbarrier_init(&empty[threadIdx.x], team_warps);
        fetched[threadIdx.x] = -1;
        fence_barrier_init();
    }
    grid_wait();
    grid_release();
    // The activations, once per CTA, every eight inputs in the order (0,4,1,5,2,6,3,7) the unpacked pairs have. Eight pieces
    // that lie together: piece j and j + 4 of a step's four groups, which is what the lanes of a warp read at a time. A lane takes
    // the piece that spreads its quarter of the warp over two lines to load and over all banks twice to store: pieces in a row
    // are stored four to a bank. Four loads are under way at a time, where a launch has one matrix to spread them over: 8 x 896 x
    // 3072 4.6 -> 4.1 us (with pieces in a row 4.25, one load at a time 4.5), 5 x 3072 x 1536 3.55 -> 3.3, 1 x 3072 x 3072 the same. In
    // the grouped form it is one, for four made 60 x 9216 x 1024 88 -> 90.
    constexpr int AT_ONCE = GROUPED ? 1 : 4;
    const uint32_t x_pairs = smem + stages * stage_bytes, x_row = stream_x_pieces(k) * 16;
    const int x_pieces = steps * STREAM_STEP_GROUPS * 8, x_items = m * x_pieces;
    for (int item0 = threadIdx.x; item0 < x_items; item0 += AT_ONCE * STREAM_THREADS) {
        uint4 v[AT_ONCE];
        uint32_t to[AT_ONCE];
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            const int item = item0 + i * STREAM_THREADS;
            if (item >= x_items) break;
            const int row = item / x_pieces, place = item - row * x_pieces;
            const int piece = (place & ~31) + (place & 1) + (place >> 4 & 1) * 2 + (place >> 1 & 7) * 4;  // input / 8
            v[i] = make_uint4(0u, 0u, 0u, 0u);  // a ragged last step is filled with zeros
            if (piece < k / 8) v[i] = __ldg(reinterpret_cast<const uint4 *>(x) + static_cast<size_t>(row) * (k / 8) + piece);
            to[i] = x_pairs + row * x_row + ((piece & ~31) + (piece & 3) * 8 + (piece >> 2 & 1) * 4 + (piece >> 3 & 3)) * 16;
        }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            if (item0 + i * STREAM_THREADS >= x_items) break;
            sts_16(to[i], make_uint4(__byte_perm(v[i].x, v[i].z, 0x5410), __byte_perm(v[i].x, v[i].z, 0x7632), __byte_perm(v[i].y, v[i].w, 0x5410), __byte_perm(v[i].y, v[i].w, 0x7632)));
        }
    }
    __syncthreads();
    if (cta_warp == STREAM_WARPS) {
        if (lane == 0) {
            int item_index = 0, local = blockIdx.x;
            uint32_t s = 0, phase = 1;
            for (int tile = local; tile < tiles; tile += step_tiles, local += step_tiles) {
                if (GROUPED)
                    while (local >= tiles_each) local -= tiles_each, ++item_index;
                if (!mbarrier_wait(&empty[s], phase, &g_status, STATUS_WAIT_EMPTY | 0xB100 | s, 64)) break;
                fetch(tile, item_index, local, s);
                if (++s == static_cast<uint32_t>(stages)) s = 0, phase ^= 1;
            }
        }
        return;
    }

    const __half2 sixty_fourth = __float2half2_rn(1.0f / 64.0f), quarter = __float2half2_rn(0.25f), two_to_9 = __float2half2_rn(512.0f), sixteen = __float2half2_rn(16.0f);
    // This warp's slice of K; HALVES: of two warps with one slice each takes one half of every group.
    const uint32_t slices = HALVES ? team_warps / 2 : team_warps, slice = HALVES ? warp >> 1 : warp, half = HALVES ? warp & 1 : 0;
    const uint32_t whole = groups / STREAM_STEP_GROUPS, first = steps * slice / slices, last = steps * (slice + 1) / slices;
    // Row r of the MMA is weight row r / 2 where r is even, 8 + r / 2 where it is odd; row r + 8 the fourth after that.
    const uint32_t weight_row = (r >> 1) + (r & 1) * 8;
    // Lane / 4 is the number of the B operand's column, an activation row. A column only ever meets its own results: a lane past
    // the last row feeds row 0 again, and what comes of it is not stored.
    const uint32_t my_x = x_pairs + (r < static_cast<uint32_t>(m) ? r : 0) * x_row + q * 16 + half * 64 + first * 512;
    const uint32_t my_codes = weight_row * row_bytes + (r & 1) * shift + q * 32 + half * 16 + first * 128;
    const uint32_t my_scales = scales_at + (weight_row * groups + q + first * STREAM_STEP_GROUPS) * 2;
    const uint32_t slice_bytes = m * STREAM_ROWS * 4;
    const uint32_t partials = x_pairs + m * x_row + team * 2 * team_warps * slice_bytes;
    const uint32_t my_partial = warp * slice_bytes + weight_row * 4 + 2 * q * (STREAM_ROWS * 4);
    const bool stores = 2 * q < static_cast<uint32_t>(m), stores_too = 2 * q + 1 < static_cast<uint32_t>(m);
    const bool sums = team_thread < m * STREAM_ROWS;
    // Team t takes the CTA's tiles t, t + teams, ...; tile i of the CTA lies in stage i modulo the number of stages.
    uint32_t s = team, phase = 0, parity = 0;
    while (s >= static_cast<uint32_t>(stages)) s -= stages, phase ^= 1;
    const int team_step = teams * step_tiles;
    int item_index = 0, local = blockIdx.x + team * step_tiles;
    bool gave_up = false;
    for (int tile = local; tile < tiles; tile += team_step, local += team_step, parity ^= 1) {
        if (GROUPED)
            while (local >= tiles_each) local -= tiles_each, ++item_index;
        const uint32_t partial = partials + parity * team_warps * slice_bytes;
        const float *to_bias = bias;
        void *to_y = y;
        if (GROUPED) to_bias = group->item[item_index].bias, to_y = group->item[item_index].y;
        const int out_row = local * STREAM_ROWS + (team_thread & 15);
        float add = 0.0f;
        if (sums && to_bias != nullptr) add = __ldg(to_bias + out_row);
        // The stage's last user may have been another team. Only once this tile has been sent for is the phase before complete,
        // and the parity of this one's unambiguous.
        const bool arrived = wait_uniform([&]() { return fetched[s] == tile; }, &g_status, STATUS_WAIT_EMPTY | 0xB000 | s, 32) &&
                             mbarrier_wait_uniform(full_u + s * 8, phase, &g_status, STATUS_WAIT_FULL | 0xB000 | s);
        const uint32_t stage = smem + s * stage_bytes;
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f}, d[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // of a group's first half, of its second
        if (arrived) {
            uint32_t at_codes = stage + my_codes, at_codes_b = at_codes + 4 * row_bytes, at_x = my_x;
            uint32_t at_scales = stage + my_scales, at_scales_b = at_scales + 8 * groups;
#pragma unroll 1
            for (uint32_t step = first; step < last; ++step, at_codes += 128, at_codes_b += 128, at_x += 512, at_scales += 8, at_scales_b += 8) {
                __half scale_a = lds_half(at_scales), scale_b = lds_half(at_scales_b);
                __half minimum_a = lds_half(at_scales + scale_bytes), minimum_b = lds_half(at_scales_b + scale_bytes);
                if (step >= whole && step * STREAM_STEP_GROUPS + q >= groups)  // past a ragged end: what was read lies in the CTA's shared memory; zeros
                    scale_a = scale_b = minimum_a = minimum_b = __ushort_as_half(0);
                uint4 code_a[2], code_b[2];
                code_a[0] = lds_16(at_codes), code_b[0] = lds_16(at_codes_b);
                if constexpr (!HALVES) code_a[1] = lds_16(at_codes + 16), code_b[1] = lds_16(at_codes_b + 16);
                const __half2 ma = __half2half2(minimum_a), mb = __half2half2(minimum_b);
                auto multiply = [&](auto unpack) {
#pragma unroll
                    for (int w = 0; w < (HALVES ? 4 : 8); ++w) {  // 8 inputs of each row per word, two MMA steps
                        const uint4 xv = lds_16(at_x + (w >> 2) * 64 + (w & 3) * 128);
                        const uint4 from_a = code_a[w >> 2], from_b = code_b[w >> 2];
                        const uint32_t a = (w & 3) == 0 ? from_a.x : (w & 3) == 1 ? from_a.y : (w & 3) == 2 ? from_a.z : from_a.w;
                        const uint32_t b = (w & 3) == 0 ? from_b.x : (w & 3) == 1 ? from_b.y : (w & 3) == 2 ? from_b.z : from_b.w;
                        uint32_t pa[4], pb[4];
                        unpack(a, b, pa, pb);
                        const uint32_t one[4] = {pa[0], pb[0], pa[1], pb[1]}, two[4] = {pa[2], pb[2], pa[3], pb[3]};
                        mma_m16n8k16(w >> 2 ? d : c, one, xv.x, xv.y);
                        mma_m16n8k16(w >> 2 ? d : c, two, xv.z, xv.w);
                    }
                };
                // scale * 2^22 is an fp16 number below 1/64, scale * 2^18 below 1/4 (a NaN fails both tests)
                const __half2 both = __halves2half2(scale_a, scale_b), magnitudes = __habs2(both);
                if (__all_sync(0xffffffffu, __hblt2(magnitudes, sixty_fourth))) {
                    const __half2 up = __hmul2(__hmul2(both, two_to_9), two_to_9), up_22 = __hmul2(up, sixteen);
                    const __half2 sa = __low2half2(up), sb = __high2half2(up), sa_22 = __low2half2(up_22), sb_22 = __high2half2(up_22);
                    multiply([&](uint32_t a, uint32_t b, uint32_t(&pa)[4], uint32_t(&pb)[4]) {
                        unpack_word<false>(a, sa_22, sa, ma, pa);
                        unpack_word<false>(b, sb_22, sb, mb, pb);
                    });
                } else if (__all_sync(0xffffffffu, __hblt2(magnitudes, quarter))) {
                    const __half2 up = __hmul2(__hmul2(both, two_to_9), two_to_9), sa = __low2half2(up), sb = __high2half2(up);
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
        if constexpr (!HALVES) {
#pragma unroll
            for (int i = 0; i < 4; ++i) c[i] += d[i];
        }
        // c[0], c[1]: MMA row r, columns 2q, 2q+1; c[2], c[3]: MMA row r + 8
        if (stores) {
            sts_float(partial + my_partial, c[0]);
            sts_float(partial + my_partial + 16, c[2]);
        }
        if (stores_too) {
            sts_float(partial + my_partial + STREAM_ROWS * 4, c[1]);
            sts_float(partial + my_partial + STREAM_ROWS * 4 + 16, c[3]);
        }
        __syncwarp();
        if (lane == 0) mbarrier_arrive_u32(empty_u + s * 8);  // this warp is done with the stage
        // The partial sums are complete. They alternate between two places: those of this tile are read below and
        // written again two tiles on, with the next tile's barrier in between.
        named_barrier_sync(1 + team, team_threads);
        gave_up |= !arrived;
        // fixed-order sum over the K slices: thread -> (activation row, weight row), so that few rows keep few warps
        if (sums) {
            for (uint32_t item = team_thread; item < slice_bytes / 4; item += team_threads) {
                float of_slice[STREAM_MAX_SLICES], of_half[STREAM_MAX_SLICES], total = 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < (HALVES ? STREAM_MAX_SLICES / 2 : STREAM_MAX_SLICES); ++i)
                    if (i < slices) {
                        of_slice[i] = lds_float(partial + (HALVES ? 2 * i : i) * slice_bytes + item * 4);
                        if constexpr (HALVES) of_half[i] = lds_float(partial + (2 * i + 1) * slice_bytes + item * 4);
                    }
#pragma unroll
                for (uint32_t i = 0; i < (HALVES ? STREAM_MAX_SLICES / 2 : STREAM_MAX_SLICES); ++i)
                    if (i < slices) total += HALVES ? of_slice[i] + of_half[i] : of_slice[i];
                total += add;
                const size_t element = static_cast<size_t>(item >> 4) * ldy + out_row;
                if (y_is_half) static_cast<__half *>(to_y)[element] = __float2half_rn(total);
                else static_cast<float *>(to_y)[element] = total;
            }
        }
        s += teams;
        while (s >= static_cast<uint32_t>(stages)) s -= stages, phase ^= 1;
    }
    // Every copy has a team that waits for it. Where a wait gave up, let the copies already issued land. (Asking the status
    // word instead is a round trip to L2 at the end of every CTA: 4080 x 4096 5.6 -> 5.9 us.)
    if (gave_up) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
}

template <bool HALVES>
__global__ void __launch_bounds__(STREAM_THREADS, 1)
gemv_stream_kernel(const __half *__restrict__ x, const uint8_t *__restrict__ codes, const __half *__restrict__ scales,
                   const __half *__restrict__ minimums, const float *__restrict__ bias, void *__restrict__ y,
                   int m, int n, int k, long long ldy, int y_is_half, int stages, int team_warps) {
    gemv_stream_body<false, HALVES>(x, codes, scales, minimums, bias, y, m, n, k, ldy, y_is_half, stages, team_warps, nullptr, 1);
}

template <bool HALVES>
__global__ void __launch_bounds__(STREAM_THREADS, 1)
gemv_stream_grouped_kernel(const __half *__restrict__ x, const __grid_constant__ StreamItems group, int count,
                           int m, int n, int k, long long ldy, int y_is_half, int stages, int team_warps) {
    gemv_stream_body<true, HALVES>(x, nullptr, nullptr, nullptr, nullptr, nullptr, m, n, k, ldy, y_is_half, stages, team_warps, &group, count);
}

}  // namespace w4a16
}  // namespace qi

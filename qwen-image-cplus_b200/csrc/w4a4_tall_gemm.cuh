// W4A4 (H256, g64) GEMM on byte-wide (E4M3) codes for many rows: one 256 x 64 output tile per CTA, two 128-row halves that
// share the weight scales. Same operator, arithmetic and bits as w4a4_pair_gemm.cuh (reference:
// qwen_image_cuda/cuda/gemm.cu:65-189).
//
// What bounds it: the fold, y += (dot * sa) * sw in two fp32 operations per output and group, 256 cycles of the fp32 pipe for
// 128 x 128 outputs and a group, and around it the fold warps' other work. The pair kernel's fold threads own 1 row x 32
// columns: 32 weight scales from shared memory for 32 outputs, and the load/store data path is busy in 457 of the 564
// cycles of such a step (ncu: l1tex__data_pipe_lsu_wavefronts), the tensor cores' operand reads 157 more. Here
//   * a fold thread owns 2 rows x 32 columns: a weight scale that it loads serves two rows (457 -> 273 wavefronts)
//   * eight fold warps with up to 208 registers a thread instead of sixteen with 96: half as many looks at barriers, hand-backs
//     and loop instructions an output (1479 -> 856 instructions per SM and step), and the dots of a whole group, 64 a
//     thread, in flight at once
//   * activation scales stand in shared memory as {sa, sa} of both rows, ready for the packed multiplies
//   * a look at a barrier is one try_wait and one vote: control flow stays uniform (a per-lane branch with the
//     reconvergence behind it took 17 instructions more), at one look per two groups
// 4096 x 9216 x 3072: 240.7 -> 198 us. Measured on the way (us): sixteen fold warps of 2 x 16 columns 216; with the next dots
// copied while the present ones are folded 232 to 240 there (register moves), 216 to 222 with eight warps; one group per
// TMEM buffer 217 to 236 (a look costs some 120 cycles of a warp's chain). Taking work away from the sixteen-warp form: no
// operand loads 211, no MMAs 201, no copies out of TMEM 191, neither of the last two 176, no arithmetic 149.
//
//   warp 0      TMA: 256 A rows and 64 B rows, 128 inputs (a slab, two groups) a stage
//   warps 1, 2  tcgen05.mma kind::f8f6f4 (M = 128, twice two K steps a group), slab by slab in turn, a TMEM buffer each
//   warp 3      scales to fp32 in shared memory, four groups a slot
//   warps 4-11  fold: 32 rows of both halves x half of the columns each
#pragma once
#include "ptx.cuh"
#include "w4a16_gemm.cuh"
#include "w4a4_pair_gemm.cuh"

namespace qi {
namespace w4a4_tall {

using w4a4_pair::arrive_u32;
using w4a4_pair::lds_pairs;
using w4a4_pair::try_wait_u32;

constexpr int HALVES = 2, HALF_ROWS = 128, BM = HALVES * HALF_ROWS, BN = 64;
constexpr int SLAB_K = 128, SLAB_GROUPS = 2, SLOT_GROUPS = 4, SLOT_SLABS = SLOT_GROUPS / SLAB_GROUPS;
// An even number of stages: an issuing warp keeps to every other one, so that the load it waits for can only be the next.
constexpr int STAGES = 4, BUFFERS = 2, SLOTS = 3;
constexpr int GROUP_COLUMNS = HALVES * BN, BUFFER_COLUMNS = SLAB_GROUPS * GROUP_COLUMNS;
constexpr int PRODUCER_WARP = 0, MMA_WARP = 1, SCALE_WARP = 3, FOLD_WARP0 = 4, FOLD_WARPS = 8, SLICES = FOLD_WARPS / 4;
constexpr int THREADS = 32 * (FOLD_WARP0 + FOLD_WARPS);
constexpr int COLUMNS = BN / SLICES;  // of a fold warp in a wide tile; 24, 16 or 8 in a narrow one
constexpr int A_BYTES = BM * SLAB_K, B_BYTES = BN * SLAB_K;
constexpr int SW_BYTES = SLOT_GROUPS * BN * 4;           // fp32 [group][column]
constexpr int SA_GROUP_BYTES = HALF_ROWS * 16, SA_BYTES = SLOT_GROUPS * SA_GROUP_BYTES;  // float4 [group][row of a half] = {sa, sa} of the upper, of the lower row
constexpr int BARRIERS = 2 * STAGES + 2 * BUFFERS + 2 * SLOTS, BARRIER_BYTES = 256;
constexpr int SMEM_BYTES = STAGES * (A_BYTES + B_BYTES) + SLOTS * (SW_BYTES + SA_BYTES) + BARRIER_BYTES + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory budget of one CTA");
static_assert(BARRIERS * 8 + 4 <= BARRIER_BYTES && BUFFERS * BUFFER_COLUMNS == 512, "barrier block; the whole of TMEM");
static_assert(STAGES % BUFFERS == 0 && SLOT_SLABS == BUFFERS, "a slab's place in its slot is its TMEM buffer");
// setmaxnreg: what the two kinds of warps hold afterwards has to be there at launch, or the kernel waits for ever.
constexpr int LAUNCH_REGISTERS = 168, CONTROL_REGISTERS = 88, FOLD_REGISTERS = 208;
static_assert(THREADS * LAUNCH_REGISTERS <= 65536 && 65536 / THREADS / 8 * 8 == LAUNCH_REGISTERS, "what __launch_bounds__ gives a thread");
static_assert(FOLD_WARP0 * CONTROL_REGISTERS + FOLD_WARPS * FOLD_REGISTERS <= THREADS / 32 * LAUNCH_REGISTERS, "setmaxnreg.inc would wait for registers that do not exist");
constexpr uint32_t AHEAD_BACKOFF_NS = 100, FOLD_BACKOFF_NS = 100, MMA_BACKOFF_NS = 32;

// The order of the tiles. Wide tiles walk down a block of `block` rows of tiles, column by column, then the next block: a
// block's activations stay in L2 while the weights pass (16384 x 3072 x 12288 reads its 201 MB of activations once instead
// of once a wave). `wide` of them come first; what would be a last, partly idle wave of the last block is cut again into tiles of `width`
// columns, as many as there are CTAs or fewer. Rows of tiles below tail_row (counted in the last block) start their narrow tiles one wide tile later.
struct Tiling {
    int tiles, wide, width;
    int tiles_m, tiles_n, block;
    int last, last_rows;  // first row of tiles of the last block, and how many it has
    int tail_row, tail_n, tail_later, tail_sooner;
};
struct TilePlace {
    int m0, n0, width;
};
__device__ __forceinline__ TilePlace place(const Tiling &t, int tile) {
    if (tile < t.wide) {
        const int in_block = t.block * t.tiles_n, first = tile / in_block * t.block, rest = tile % in_block;
        const int rows = min(t.block, t.tiles_m - first);
        return {(first + rest % rows) * BM, rest / rows * BN, BN};
    }
    int narrow = tile - t.wide;
    const int later = t.tail_row * t.tail_later;
    if (narrow < later) return {(t.last + narrow % t.tail_row) * BM, t.tail_n + BN + narrow / t.tail_row * t.width, t.width};
    narrow -= later;
    const int rows = t.last_rows - t.tail_row;
    return {(t.last + t.tail_row + narrow % rows) * BM, t.tail_n + narrow / rows * t.width, t.width};
}

// A look at a barrier by a converged warp: the vote's answer is the same in every lane, and nothing diverges.
__device__ __noinline__ bool look_slow(uint32_t barrier, uint32_t parity, uint32_t code) {
    return mbarrier_wait_uniform(barrier, parity, &g_status, code, FOLD_BACKOFF_NS);
}
__device__ __forceinline__ bool look(uint32_t barrier, uint32_t parity, uint32_t code) {
    return __all_sync(0xffffffffu, try_wait_u32(barrier, parity)) || look_slow(barrier, parity, code);
}

__device__ __forceinline__ void tmem_load_32x8(uint32_t address, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(address) : "memory");
}
template <int WIDTH>
__device__ __forceinline__ void load_dots(uint32_t address, uint32_t (&r)[WIDTH]) {
    if constexpr (WIDTH == 32) tmem_load_32x32(address, r);
    if constexpr (WIDTH == 16 || WIDTH == 24) tmem_load_32x16(address, reinterpret_cast<uint32_t(&)[16]>(r));
    if constexpr (WIDTH == 8 || WIDTH == 24) tmem_load_32x8(address + WIDTH - 8, r + WIDTH - 8);
}
// The wait for all copies out of TMEM, with their registers tied to it.
template <int WIDTH>
__device__ __forceinline__ void wait_dots(uint32_t (&r)[HALVES][WIDTH]) {
    tmem_load_wait();
#pragma unroll
    for (int half = 0; half < HALVES; ++half)
#pragma unroll
        for (int j = 0; j < WIDTH; j += 8)
            asm volatile("" : "+r"(r[half][j]), "+r"(r[half][j + 1]), "+r"(r[half][j + 2]), "+r"(r[half][j + 3]), "+r"(r[half][j + 4]), "+r"(r[half][j + 5]),
                         "+r"(r[half][j + 6]), "+r"(r[half][j + 7])::"memory");
}

struct FoldState {
    uint32_t tmem, sw, sa;  // of this warp's columns, of this thread's rows
    uint32_t dot_full, dot_empty, scale_full, scale_empty;
    uint32_t slot, slot_phase, dot_phase;
};

// One tile's 2 rows x WIDTH columns of this thread, from n0 on. False when a wait ran out of time.
template <int WIDTH>
__device__ __forceinline__ bool fold_tile(FoldState &f, int row, int n0, int slots, const float *__restrict__ bias, void *__restrict__ y, const GemmShape &shape, int lane) {
    uint64_t acc[HALVES][WIDTH / 2];
#pragma unroll
    for (int j = 0; j < WIDTH; ++j) acc[j % HALVES][j / HALVES] = 0;
#pragma unroll 1
    for (int ks = 0; ks < slots; ++ks) {
        if (!look(f.scale_full + f.slot * 8, f.slot_phase, STATUS_WAIT_READY | 0xA000 | f.slot)) return false;
        const uint32_t sw = f.sw + f.slot * SW_BYTES, sa = f.sa + f.slot * SA_BYTES;
#pragma unroll
        for (int g = 0; g < SLOT_GROUPS; ++g) {
            const int buffer = g / SLAB_GROUPS;
            if (g % SLAB_GROUPS == 0) {
                if (!look(f.dot_full + buffer * 8, f.dot_phase, STATUS_WAIT_TMEM_FULL | 0xA000 | buffer)) return false;
                tcgen05_fence_after();
            }
            uint32_t dots[HALVES][WIDTH];
#pragma unroll
            for (int half = 0; half < HALVES; ++half) load_dots<WIDTH>(f.tmem + g * GROUP_COLUMNS + half * BN, dots[half]);
            const ulonglong2 sa2 = lds_pairs(sa + g * SA_GROUP_BYTES);
            wait_dots<WIDTH>(dots);
            if (g % SLAB_GROUPS == SLAB_GROUPS - 1) {  // the whole warp's dots of both groups are in registers or folded
                tcgen05_fence_before();
                __syncwarp();  // every lane's copies are ordered before the one arrival
                if (lane == 0) arrive_u32(f.dot_empty + buffer * 8);
            }
#pragma unroll
            for (int q = 0; q < WIDTH / 4; ++q) {  // dot * sa and sa * sw are exact: rounded once, in the fused multiply-add
                const ulonglong2 sw4 = lds_pairs(sw + (g * BN + 4 * q) * 4);
                acc[0][2 * q] = fma_f32x2(mul_f32x2(pack_u32x2(dots[0][4 * q], dots[0][4 * q + 1]), sa2.x), sw4.x, acc[0][2 * q]);
                acc[0][2 * q + 1] = fma_f32x2(mul_f32x2(pack_u32x2(dots[0][4 * q + 2], dots[0][4 * q + 3]), sa2.x), sw4.y, acc[0][2 * q + 1]);
                acc[1][2 * q] = fma_f32x2(mul_f32x2(pack_u32x2(dots[1][4 * q], dots[1][4 * q + 1]), sa2.y), sw4.x, acc[1][2 * q]);
                acc[1][2 * q + 1] = fma_f32x2(mul_f32x2(pack_u32x2(dots[1][4 * q + 2], dots[1][4 * q + 3]), sa2.y), sw4.y, acc[1][2 * q + 1]);
            }
        }
        f.dot_phase ^= 1;
        __syncwarp();
        if (lane == 0) arrive_u32(f.scale_empty + f.slot * 8);
        if (++f.slot == SLOTS) f.slot = 0, f.slot_phase ^= 1;
    }
    // n is a multiple of 32 and n0 of 8: eight columns exist or do not. Whole 32-byte sectors where the rows are aligned for them.
    const bool sectors = WIDTH % 16 == 0 && (n0 & 15) == 0 && (reinterpret_cast<uintptr_t>(y) & 31) == 0 && shape.ldy % (shape.y_is_half ? 16 : 8) == 0;
#pragma unroll
    for (int half = 0; half < HALVES; ++half) {
        if (row + half * HALF_ROWS >= shape.m) break;
        const size_t element = static_cast<size_t>(row + half * HALF_ROWS) * shape.ldy + n0;
#pragma unroll
        for (int j = 0; j < WIDTH; j += 16) {
            if (n0 + j >= shape.n) break;
            constexpr int LAST = WIDTH % 16 == 0 ? 16 : 8;
            const int count = j + 16 <= WIDTH && n0 + j + 16 <= shape.n ? 16 : 8;  // columns that exist
            float out[16];
#pragma unroll
            for (int i = 0; i < (j + 16 <= WIDTH ? 16 : LAST); i += 2) unpack_f32x2(acc[half][(j + i) / 2], out[i], out[i + 1]);
            if (bias != nullptr) {
#pragma unroll
                for (int i = 0; i < (j + 16 <= WIDTH ? 16 : LAST); ++i)
                    if (i < count) out[i] += __ldg(bias + n0 + j + i);
            }
            if (shape.y_is_half) {
                uint32_t h[8];
#pragma unroll
                for (int i = 0; i < (j + 16 <= WIDTH ? 8 : LAST / 2); ++i) {
                    const __half2 pair = __floats2half2_rn(out[2 * i], out[2 * i + 1]);
                    h[i] = *reinterpret_cast<const uint32_t *>(&pair);
                }
                __half *target = static_cast<__half *>(y) + element + j;
                if (sectors && count == 16) st_global_v8(target, h);
                else {
                    *reinterpret_cast<uint4 *>(target) = make_uint4(h[0], h[1], h[2], h[3]);
                    if (j + 16 <= WIDTH && count == 16) *reinterpret_cast<uint4 *>(target + 8) = make_uint4(h[4], h[5], h[6], h[7]);
                }
            } else {
                float *target = static_cast<float *>(y) + element + j;
#pragma unroll
                for (int i = 0; i < (j + 16 <= WIDTH ? 16 : LAST); i += 8) {
                    if (i >= count) break;
                    if (sectors) st_global_v8(target + i, reinterpret_cast<const uint32_t(&)[8]>(out[i]));
                    else {
                        *reinterpret_cast<float4 *>(target + i) = make_float4(out[i], out[i + 1], out[i + 2], out[i + 3]);
                        *reinterpret_cast<float4 *>(target + i + 4) = make_float4(out[i + 4], out[i + 5], out[i + 6], out[i + 7]);
                    }
                }
            }
        }
    }
    return true;
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
            const __half *__restrict__ a_scales, const __half *__restrict__ w_scales,
            const float *__restrict__ bias, void *__restrict__ y, const GemmShape shape, const __grid_constant__ Tiling tiling) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float *sw_slots = reinterpret_cast<float *>(smem + STAGES * (A_BYTES + B_BYTES)), *sa_slots = sw_slots + SLOTS * SW_BYTES / 4;
    uint64_t *barriers = reinterpret_cast<uint64_t *>(sa_slots + SLOTS * SA_BYTES / 4);
    const uint32_t tile_a = smem_u32(smem), tile_b = tile_a + STAGES * A_BYTES;
    const uint32_t full = smem_u32(barriers), empty = full + 8 * STAGES, dot_full = empty + 8 * STAGES, dot_empty = dot_full + 8 * BUFFERS;
    const uint32_t scale_full = dot_empty + 8 * BUFFERS, scale_empty = scale_full + 8 * SLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(barriers + BARRIERS);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int slabs = shape.k / SLAB_K, slots = shape.k / (64 * SLOT_GROUPS), step = static_cast<int>(gridDim.x);

    if (threadIdx.x == 0) {
        for (int i = 0; i < BARRIERS; ++i) {
            const int dot_empty0 = 2 * STAGES + BUFFERS, scale_empty0 = 2 * STAGES + 2 * BUFFERS + SLOTS;
            mbarrier_init(barriers + i, (i >= dot_empty0 && i < dot_empty0 + BUFFERS) || i >= scale_empty0 ? FOLD_WARPS : 1);
        }
        fence_barrier_init();
    }
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, BUFFERS * BUFFER_COLUMNS);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    grid_wait();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < FOLD_WARP0) {
        setmaxnreg_dec<CONTROL_REGISTERS>();
        if (warp == PRODUCER_WARP) {
            if (lane == 0) {
                prefetch_tensormap(&map_a);
                prefetch_tensormap(&map_w);
                uint32_t s = 0, phase = 1;
                bool alive = true;
                for (int tile = blockIdx.x; tile < tiling.tiles && alive; tile += step) {
                    const TilePlace at = place(tiling, tile);
                    for (int slab = 0; slab < slabs; ++slab) {
                        if (!mbarrier_wait(barriers + STAGES + s, phase, &g_status, STATUS_WAIT_EMPTY | 0xA000 | s, AHEAD_BACKOFF_NS)) { alive = false; break; }
                        mbarrier_arrive_expect_tx_u32(full + s * 8, A_BYTES + B_BYTES);
                        tma_load_2d_u32(tile_a + s * A_BYTES, &map_a, full + s * 8, slab * SLAB_K, at.m0);
                        tma_load_2d_u32(tile_b + s * B_BYTES, &map_w, full + s * 8, slab * SLAB_K, at.n0);  // 64 rows, of a narrow tile too
                        if (++s == STAGES) s = 0, phase ^= 1;
                    }
                }
            }
        } else if (warp == MMA_WARP || warp == MMA_WARP + 1) {
            const uint32_t mine = static_cast<uint32_t>(warp - MMA_WARP);
            const uint64_t a_first = umma_desc_k_sw128(tile_a), b_first = umma_desc_k_sw128(tile_b);
            const uint32_t accumulator = tmem_base + mine * BUFFER_COLUMNS, my_full = dot_full + mine * 8, my_empty = dot_empty + mine * 8;
            uint32_t s = mine, phase = 0, buffer_phase = 1;
            bool alive = true;
            for (int tile = blockIdx.x; tile < tiling.tiles && alive; tile += step) {
                const uint32_t idesc = umma_idesc_e4m3_f32(HALF_ROWS, 0) | (static_cast<uint32_t>(tile < tiling.wide ? BN : tiling.width) >> 3 << 17);
                for (int slab = mine; slab < slabs; slab += BUFFERS) {  // k is a multiple of 256: both warps have as many
                    if (!mbarrier_wait_uniform2(full + s * 8, phase, my_empty, buffer_phase, &g_status, STATUS_WAIT_TMEM_EMPTY | 0xA000 | s, MMA_BACKOFF_NS)) { alive = false; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint64_t a_desc = a_first + s * (A_BYTES >> 4), b_desc = b_first + s * (B_BYTES >> 4);
#pragma unroll
                        for (int g = 0; g < SLAB_GROUPS; ++g)
#pragma unroll
                            for (int half = 0; half < HALVES; ++half)
#pragma unroll
                                for (int kk = 0; kk < 2; ++kk)
                                    umma_f8(accumulator + g * GROUP_COLUMNS + half * BN, a_desc + half * (HALF_ROWS * SLAB_K >> 4) + g * 4 + kk * 2, b_desc + g * 4 + kk * 2, idesc, kk);
                        tcgen05_commit_u32(my_full);
                        tcgen05_commit_u32(empty + s * 8);
                    }
                    __syncwarp();
                    buffer_phase ^= 1;
                    s += BUFFERS;
                    if (s >= STAGES) s -= STAGES, phase ^= 1;
                }
            }
        } else if (warp == SCALE_WARP) {
            // A lane's columns and rows, eight groups (sixteen bytes) each: two slots. They are asked for once the two before are
            // written, which the fold warps still need for two slots' time. Four groups at a time, a row's 32-byte sector was
            // asked for four times, and where the rows of a tile are more than L1 keeps beside 190 KB of shared memory, from L2 each
            // time (without any of these loads 4096 x 3072 x 12288 took 288 us instead of 303): 4096 x 3072 x 12288 305 -> 297 us,
            // 1024 x 12288 x 4096 108 -> 105, 4096 x 9216 x 3072 the same. Where rows do not begin on sixteen bytes (an odd number of slots)
            // each half is a load of its own, and 62 such GEMMs take 0.7 percent longer than with four groups at a time, up to 1.6 (1995 x 2976 x 3328
            // 42.3 -> 42.9; one, 970 x 1504 x 5376, 3). A loop of its own for them made all shapes 1 to 2 percent slower, one loop of single slots
            // for both 1 to 5: the fold warps feel every instruction here. Rows and columns that do not exist take the last one's: nothing
            // reads what becomes of them.
            constexpr int SW_ITEMS = BN / 32, SA_ITEMS = BM / 32, ITEMS = SW_ITEMS + SA_ITEMS, LOWER = SA_ITEMS / HALVES;
            const bool whole = slots % 2 == 0 && ((reinterpret_cast<uintptr_t>(w_scales) | reinterpret_cast<uintptr_t>(a_scales)) & 15) == 0;
            uint32_t slot = 0, phase = 1;
            bool alive = true;
            for (int tile = blockIdx.x; tile < tiling.tiles && alive; tile += step) {
                const TilePlace at = place(tiling, tile);
                uint32_t from[ITEMS];  // in slots
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    const int index = i < SW_ITEMS ? min(at.n0 + i * 32 + lane, shape.n - 1) : min(at.m0 + (i - SW_ITEMS) * 32 + lane, shape.m - 1);
                    from[i] = static_cast<uint32_t>(index) * slots;
                }
                for (int ks = 0; ks < slots && alive; ks += 2) {
                    uint4 next[ITEMS];
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i) {
                        const uint2 *source = reinterpret_cast<const uint2 *>(i < SW_ITEMS ? w_scales : a_scales) + from[i] + ks;
                        if (whole) {
                            next[i] = __ldg(reinterpret_cast<const uint4 *>(source));
                        } else {
                            const uint2 first = __ldg(source), second = ks + 1 < slots ? __ldg(source + 1) : make_uint2(0u, 0u);
                            next[i] = make_uint4(first.x, first.y, second.x, second.y);
                        }
                    }
#pragma unroll
                    for (int sub = 0; sub < 2; ++sub) {
                        if (ks + sub >= slots) break;
                        if (!mbarrier_wait_uniform(scale_empty + slot * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0xA100 | slot, AHEAD_BACKOFF_NS)) { alive = false; break; }
#pragma unroll
                        for (int i = 0; i < SW_ITEMS; ++i) {
                            const uint32_t raw_low = sub ? next[i].z : next[i].x, raw_high = sub ? next[i].w : next[i].y;
                            const float2 low = __half22float2(*reinterpret_cast<const __half2 *>(&raw_low)), high = __half22float2(*reinterpret_cast<const __half2 *>(&raw_high));
                            float *to = sw_slots + slot * (SW_BYTES / 4) + i * 32 + lane;
                            to[0] = low.x, to[BN] = low.y, to[2 * BN] = high.x, to[3 * BN] = high.y;
                        }
#pragma unroll
                        for (int i = 0; i < LOWER; ++i) {
                            const uint4 upper = next[SW_ITEMS + i], lower = next[SW_ITEMS + LOWER + i];
                            float4 *to = reinterpret_cast<float4 *>(sa_slots + slot * (SA_BYTES / 4)) + i * 32 + lane;
#pragma unroll
                            for (int pair = 0; pair < 2; ++pair) {
                                const uint32_t raw_upper = sub ? (pair ? upper.w : upper.z) : pair ? upper.y : upper.x, raw_lower = sub ? (pair ? lower.w : lower.z) : pair ? lower.y : lower.x;
                                const float2 u = __half22float2(*reinterpret_cast<const __half2 *>(&raw_upper)), l = __half22float2(*reinterpret_cast<const __half2 *>(&raw_lower));
                                to[2 * pair * HALF_ROWS] = make_float4(u.x, u.x, l.x, l.x);
                                to[(2 * pair + 1) * HALF_ROWS] = make_float4(u.y, u.y, l.y, l.y);
                            }
                        }
                        __syncwarp();
                        if (lane == 0) mbarrier_arrive_u32(scale_full + slot * 8);
                        if (++slot == SLOTS) slot = 0, phase ^= 1;
                    }
                }
            }
        }
    } else {
        setmaxnreg_inc<FOLD_REGISTERS>();
        // The hardware ties a warp to the TMEM lanes 32 * (warp % 4).
        const int quadrant = warp & 3, slice = (warp - FOLD_WARP0) >> 2;
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quadrant * 32) << 16), sw_first = smem_u32(sw_slots);
        FoldState f = {0, 0, smem_u32(sa_slots) + (quadrant * 32 + lane) * 16, dot_full, dot_empty, scale_full, scale_empty, 0, 0, 0};
        for (int tile = blockIdx.x; tile < tiling.tiles; tile += step) {
            const TilePlace at = place(tiling, tile);
            const int row = at.m0 + quadrant * 32 + lane, columns = at.width / SLICES, first = slice * columns, n0 = at.n0 + first;
            f.tmem = tmem_lane + first;
            f.sw = sw_first + first * 4;
            bool alive;
            // the wide tiles' loop last: first, the same instructions took up to a percent longer
            if (columns == 8) alive = fold_tile<8>(f, row, n0, slots, bias, y, shape, lane);
            else if (columns == 16) alive = fold_tile<16>(f, row, n0, slots, bias, y, shape, lane);
            else if (columns == 24) alive = fold_tile<24>(f, row, n0, slots, bias, y, shape, lane);
            else alive = fold_tile<32>(f, row, n0, slots, bias, y, shape, lane);
            if (!alive) break;
            __syncwarp();  // rows that do not exist left the stores early
        }
        tmem_load_wait();  // nothing of this warp may still be in flight at teardown
    }

    tcgen05_fence_before();
    __syncthreads();
    if (*reinterpret_cast<volatile uint32_t *>(&g_status) != 0) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);  // let bulk copies already issued land
    }
    if (warp == MMA_WARP) {
        __syncwarp();
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, BUFFERS * BUFFER_COLUMNS);
    }
}

}  // namespace w4a4_tall
}  // namespace qi

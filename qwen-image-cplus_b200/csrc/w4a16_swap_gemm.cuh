// W4A16 g64 dequant-GEMM with the operands' roles exchanged, for few to some thousand activation rows: the 128 rows of
// the tensor core's first operand are WEIGHT rows, unpacked straight into TMEM, and the activations are its second
// operand, whose extent N may be any multiple of 16 up to 256. Same operator and unpacking as w4a16_gemm.cuh
// (reference: qwen_image_cuda/cuda/gemm.cu:191-268).
//
// What bounds such shapes is not arithmetic: 77 x 12288 x 3072 has 48 tiles of 256 x 256, each half empty, on 148 SMs,
// and every one walks the whole of K alone. Here a tile is 128 weight rows x `columns` activation rows (77 -> 80: no
// padding to 128 or 256), and the CTAs of a cluster (1 to 8) share a tile by splitting K: each leaves a float32 partial
// tile in its shared memory and the cluster sums them through distributed shared memory in a fixed order. No workspace,
// no atomics, the same bits on every run.
//
// Per step of 128 inputs (two quantisation groups):
//   warp 0      TMA: the activations' tile (128-byte swizzled, K-major, two boxes of 64 inputs)
//   warp 2      TMA: the codes, 128 bytes of a row (two steps) at a time
//   warps 4-19  four groups of four, steps in turn: a thread unpacks 128 codes of one weight row and stores them into its
//               TMEM lane (tcgen05.st), where the tensor core reads them as its first operand: the unpacked weights
//               never pass through shared memory
//   warps 1, 3  tcgen05.mma kind::f16 with A in TMEM (M = 128, N = columns, K = 16) x 8; up to 128 columns the two take
//               the steps in turn, each into an accumulator of its own, above that warp 1 issues all
// then the unpack warps: accumulator -> bias -> y, or where CTAs share the tile accumulator -> shared memory of the CTA that
// sums the row, and all warps: sum over the cluster, bias, store (rows of y contiguous per warp).
#pragma once
#include "ptx.cuh"
#include "w4a16_gemm.cuh"

namespace qi {
namespace w4a16_swap {

constexpr int BK = 128, BN = 128;         // inputs per step: two quantisation groups; weight rows of a tile
constexpr int MAX_COLUMNS = 256, MAX_STAGES = 8, MAX_SPLIT = 8;
constexpr int PRODUCER_WARP = 0, MMA_WARP = 1, CODE_WARP = 2, SECOND_MMA_WARP = 3, UNPACK_WARP0 = 4;
constexpr int UNPACK_GROUPS = 4, UNPACK_WARPS = 4 * UNPACK_GROUPS;  // a group: one warp per 32 TMEM lanes; groups take the steps in turn
constexpr int THREADS = 128 + 32 * UNPACK_WARPS;
constexpr int A_SLOTS = 4, A_COLUMNS = BK / 2;  // TMEM columns of one unpacked step: two fp16 each
constexpr int TMEM_COLUMNS = 512;
static_assert(MAX_COLUMNS + A_SLOTS * A_COLUMNS <= TMEM_COLUMNS, "accumulator and unpacked steps");
static_assert(A_SLOTS % UNPACK_GROUPS == 0, "a group keeps to its own slots");
constexpr int TWO_ISSUERS_COLUMNS = 128;  // widest tile of which two accumulators fit
static_assert(2 * TWO_ISSUERS_COLUMNS + A_SLOTS * A_COLUMNS <= TMEM_COLUMNS, "two accumulators and unpacked steps");
__host__ __device__ constexpr int issuers_of(int columns) { return columns <= TWO_ISSUERS_COLUMNS ? 2 : 1; }
constexpr int CODE_STEPS = 2, MAX_CODE_STAGES = 6;  // steps of codes fetched together: 128 bytes of a row; chunks in flight
constexpr int CODE_BYTES = BN * CODE_STEPS * (BK / 2);
constexpr int CODE_READERS = CODE_STEPS * 4;    // warps that read a chunk: one group per step
static_assert(UNPACK_GROUPS % CODE_STEPS == 0, "a group's next step is in a chunk a whole number of chunks on");
constexpr int BARRIER_BYTES = 512;
static_assert((2 * MAX_STAGES + 2 * MAX_CODE_STAGES + A_SLOTS + 1) * 8 + 4 <= BARRIER_BYTES, "barrier block");
constexpr uint32_t AHEAD_BACKOFF_NS = 100, UNPACK_BACKOFF_NS = 20;  // pauses between polls: a polling warp takes issue slots

struct Plan {
    int columns;   // activation rows of a tile, a multiple of 16
    int split;     // CTAs of a cluster, each with its share of K
    int stages, code_stages;
};
__host__ __device__ constexpr int stage_bytes(int columns) { return columns * BK * 2; }
__host__ __device__ constexpr int tile_bytes(int columns, int stages, int code_stages) {  // the stages, later the partial tile
    const int loads = stages * stage_bytes(columns) + code_stages * CODE_BYTES, partial = (columns + MAX_SPLIT) * BN * 4;
    return loads > partial ? loads : partial;
}
__host__ __device__ constexpr int smem_bytes(int columns, int stages, int code_stages) { return tile_bytes(columns, stages, code_stages) + BARRIER_BYTES + 1024; }

// How shared memory is divided for a width: at least two chunks of codes; more of them, before more of the activations, as
// long as four stages of those fit.
// Two lengths are left out. A wait asks for the parity of a phase, and passes at once where the phase BEFORE the one in
// front of it is still open: whoever waits for a stage's next load must know that the last one has landed.
//   * Codes: a group reads every second chunk. In a ring of two the last load was its own; in a ring of four or more the
//     slot it filled before was free of the MMAs of eight steps ago, which had read it. In a ring of three nothing says so.
//   * Activations: of two issuers each takes every second step, and knows that of its own steps only: an even ring.
struct SmemPlan {
    int stages, code_stages, bytes;
};
__host__ __device__ constexpr SmemPlan smem_plan(int columns) {
    const int room = 232448 - BARRIER_BYTES - 1024;
    int code_stages = (room - 4 * stage_bytes(columns)) / CODE_BYTES;
    code_stages = code_stages < 4 ? 2 : code_stages > MAX_CODE_STAGES ? MAX_CODE_STAGES : code_stages;
    int stages = (room - code_stages * CODE_BYTES) / stage_bytes(columns);
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    if (issuers_of(columns) == 2) stages = stages / 2 * 2;
    // One CTA per SM, always: it takes all of TMEM, and a second would wait for it while its cluster waits for the second (grid_release()).
    const int bytes = smem_bytes(columns, stages, code_stages);
    return {stages, code_stages, bytes < ONE_CTA_SMEM ? ONE_CTA_SMEM : bytes};
}
constexpr bool smem_plans_are_sound() {
    for (int columns = 16; columns <= MAX_COLUMNS; columns += 16) {
        const SmemPlan plan = smem_plan(columns);
        if (plan.bytes > 232448 || plan.stages < 3 || plan.stages > MAX_STAGES || plan.code_stages < 2 || plan.code_stages == 3 || plan.code_stages > MAX_CODE_STAGES) return false;
        if (issuers_of(columns) == 2 && (plan.stages < A_SLOTS || plan.stages % 2 != 0)) return false;
    }
    return true;
}
static_assert(smem_plans_are_sound(), "shared memory of every width");

// 32 registers into this thread's TMEM lane, 32 adjacent columns.
__device__ __forceinline__ void tmem_store_32x32(uint32_t address, const uint4 (&v)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(address),
        "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w), "r"(v[2].x),
        "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w), "r"(v[4].x), "r"(v[4].y),
        "r"(v[4].z), "r"(v[4].w), "r"(v[5].x), "r"(v[5].y), "r"(v[5].z), "r"(v[5].w), "r"(v[6].x), "r"(v[6].y), "r"(v[6].z),
        "r"(v[6].w), "r"(v[7].x), "r"(v[7].y), "r"(v[7].z), "r"(v[7].w)
        : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem]^T
__device__ __forceinline__ void umma_f16_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void st_cluster_f32(uint32_t address, float value) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(address), "f"(value) : "memory");
}

// PAIRED: the scales of a step's two groups can be read with one 4-byte load (rows start 4-byte aligned).
template <bool PAIRED>
__device__ __forceinline__ uint32_t load_scale_pair(const __half *row, int group, int groups, bool inside) {
    if (!inside || group >= groups) return 0u;
    if (PAIRED) return __ldg(reinterpret_cast<const uint32_t *>(row + group));
    const uint32_t low = __half_as_ushort(__ldg(row + group)), high = group + 1 < groups ? __half_as_ushort(__ldg(row + group + 1)) : 0u;
    return low | high << 16;
}

// Both groups of a step of one weight row (64 bytes of codes, a pair of scales and minimums) into 64 TMEM columns.
// `ready` is called once before the first store.
template <typename Ready>
__device__ __forceinline__ void unpack_step(const uint8_t *codes, int piece, int swizzle, uint32_t scale, uint32_t minimum, uint32_t tmem, Ready ready) {
    uint4 packed[2][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) packed[j >> 1][j & 1] = *reinterpret_cast<const uint4 *>(codes + (((piece + j) ^ swizzle) << 4));
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const uint32_t pick = g == 0 ? 0x1010u : 0x3232u;
        const uint32_t scale2 = __byte_perm(scale, 0u, pick), minimum2 = __byte_perm(minimum, 0u, pick);
        uint4 out[8];
        w4a16::unpack64(packed[g], *reinterpret_cast<const __half2 *>(&scale2), *reinterpret_cast<const __half2 *>(&minimum2), out);
        if (g == 0) ready();
        tmem_store_32x32(tmem + g * 32, out);
    }
    tmem_store_wait();
}

template <bool PAIRED>
__global__ void __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_codes,
            const __half *__restrict__ scales, const __half *__restrict__ minimums,
            const float *__restrict__ bias, void *__restrict__ y, const GemmShape shape, const Plan plan) {
    extern __shared__ uint8_t smem_raw[];
    // the same offsets in every CTA of the cluster: the dynamic shared window starts at the same address in each
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int columns = plan.columns, share = (plan.columns + plan.split - 1) / plan.split, stages = plan.stages, code_stages = plan.code_stages, split = plan.split, half_bytes = columns * 128, x_bytes = 2 * half_bytes;
    uint8_t *smem_x = smem, *smem_c = smem + stages * x_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + tile_bytes(columns, stages, code_stages));
    uint64_t *step_done = full + MAX_STAGES;  // a ring: one commit says that a step's stage and its slot are free
    uint64_t *code_full = step_done + MAX_STAGES;
    uint64_t *code_empty = code_full + MAX_CODE_STAGES;
    uint64_t *a_ready = code_empty + MAX_CODE_STAGES;
    uint64_t *done = a_ready + A_SLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = static_cast<int>(blockIdx.x) % split, tile = static_cast<int>(blockIdx.x) / split;
    const int tiles_n = (shape.n + BN - 1) / BN, groups = shape.k / 64, k_steps = (groups + 1) / 2;
    const int n0 = (tile % tiles_n) * BN, m0 = (tile / tiles_n) * columns;
    // The ring is as long as the longer of the two that wait on it, the stages of activations and the slots of unpacked
    // weights, and even where there are two issuers, so that a barrier belongs to one of them: it then completes for a later
    // step only after both that wait on it have passed the earlier one.
    const int issuers = issuers_of(columns), ring = stages >= A_SLOTS ? stages : A_SLOTS;
    const int first = k_steps * rank / split, steps = k_steps * (rank + 1) / split - first;  // this CTA's share of K
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) mbarrier_init(&full[s], 1);
        for (int s = 0; s < ring; ++s) mbarrier_init(&step_done[s], 1);
        for (int s = 0; s < code_stages; ++s) {
            mbarrier_init(&code_full[s], 1);
            mbarrier_init(&code_empty[s], CODE_READERS);
        }
        for (int s = 0; s < A_SLOTS; ++s) mbarrier_init(&a_ready[s], 4);
        mbarrier_init(done, steps < issuers ? steps : issuers);
        fence_barrier_init();
    }
    if (warp == PRODUCER_WARP && elect_one()) prefetch_tensormap(&map_x);
    if (warp == CODE_WARP && elect_one()) prefetch_tensormap(&map_codes);
    // TMEM too before the wait. Whatever holds it on this SM can end without this kernel: see grid_release().
    if (warp == MMA_WARP) {
        tmem_alloc(tmem_slot, TMEM_COLUMNS);
        tmem_relinquish();
        grid_release();  // not before this CTA has its TMEM
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    grid_wait();
    bool alive = true;
    float own_bias = 0.0f;  // one CTA to a tile: of this thread's weight row

    // The single-threaded roles run as converged warps with one elected lane: their addresses and descriptors live in
    // uniform registers; a diverged thread takes several times as long for the same few instructions.
    if (warp == PRODUCER_WARP) {
        const uint32_t full_u = smem_u32(full), done_u = smem_u32(step_done), x_u = smem_u32(smem_x);
        uint32_t s = 0;
        int before = -1, before_phase = 0;  // the step that had the stage before
        for (int step = 0; step < steps; ++step) {
            if (step >= stages) {
                if (++before == ring) before = 0, before_phase ^= 1;
                if (!mbarrier_wait_uniform(done_u + before * 8, before_phase, &g_status, STATUS_WAIT_EMPTY | 0x8000 | s, AHEAD_BACKOFF_NS)) break;
            }
            if (elect_one()) {
                mbarrier_arrive_expect_tx_u32(full_u + s * 8, x_bytes);
                tma_load_2d_u32(x_u + s * x_bytes, &map_x, full_u + s * 8, (first + step) * BK, m0);
                tma_load_2d_u32(x_u + s * x_bytes + half_bytes, &map_x, full_u + s * 8, (first + step) * BK + 64, m0);
            }
            __syncwarp();
            if (++s == static_cast<uint32_t>(stages)) s = 0;
        }
    } else if (warp == CODE_WARP) {
        const uint32_t full_u = smem_u32(code_full), empty_u = smem_u32(code_empty), c_u = smem_u32(smem_c);
        uint32_t s = 0, phase = 1;
        for (int step = 0; step < steps; step += CODE_STEPS) {
            if (!mbarrier_wait_uniform(empty_u + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0x8200 | s, AHEAD_BACKOFF_NS)) break;
            if (elect_one()) {
                mbarrier_arrive_expect_tx_u32(full_u + s * 8, CODE_BYTES);
                tma_load_2d_u32(c_u + s * CODE_BYTES, &map_codes, full_u + s * 8, (first + step) * (BK / 2), n0);
            }
            __syncwarp();
            if (++s == static_cast<uint32_t>(code_stages)) s = 0, phase ^= 1;
        }
    } else if (warp == MMA_WARP || warp == SECOND_MMA_WARP) {
        // A step's waits, eight MMAs and commit take a warp some 600 cycles, the tensor cores four per column: up to 128
        // columns two warps take the steps in turn, each into an accumulator of its own. Only the MMAs of ONE thread are sure
        // to reach an accumulator in the order they were issued in; two warps on one accumulator, with a token that passed
        // the turn, gave sums in another order from run to run. One warp for all: 77 x 12288 x 3072 12.4 -> 13.8 us.
        const uint32_t mine = warp == MMA_WARP ? 0 : 1;
        const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + (TMEM_COLUMNS - A_SLOTS * A_COLUMNS), accumulator = tmem_base + mine * TWO_ISSUERS_COLUMNS;
        const uint32_t idesc = umma_idesc_f16_f32(BN, 0) | (static_cast<uint32_t>(columns >> 3) << 17);
        const uint32_t full_u = smem_u32(full), step_done_u = smem_u32(step_done), a_ready_u = smem_u32(a_ready), done_u = smem_u32(done);
        const uint64_t b_first = umma_desc_k_sw128(smem_u32(smem_x));
        uint32_t s = mine, phase = 0, slot = mine, slot_phase = 0, at = mine;
        for (int step = mine < static_cast<uint32_t>(issuers) ? static_cast<int>(mine) : steps; step < steps; step += issuers) {
            if (!mbarrier_wait_uniform2(full_u + s * 8, phase, a_ready_u + slot * 8, slot_phase, &g_status, STATUS_WAIT_READY | 0x8000 | s)) break;
            tcgen05_fence_after();
            if (elect_one()) {
                const uint64_t b_desc = b_first + s * (x_bytes >> 4);
                const uint32_t a = tmem_a + slot * A_COLUMNS;
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk)
                    umma_f16_a_tmem(accumulator, a + kk * 8, b_desc + (kk >> 2) * (half_bytes >> 4) + (kk & 3) * 2, idesc, (step >= issuers || kk != 0) ? 1u : 0u);
                tcgen05_commit_u32(step + issuers >= steps ? done_u : step_done_u + at * 8);  // nobody waits for an issuer's last step
            }
            __syncwarp();
            s += issuers, slot += issuers, at += issuers;
            if (s >= static_cast<uint32_t>(stages)) s -= stages, phase ^= 1;
            if (slot >= A_SLOTS) slot -= A_SLOTS, slot_phase ^= 1;
            if (at >= static_cast<uint32_t>(ring)) at -= ring;
        }
    } else if (warp >= UNPACK_WARP0) {
        const int quadrant = warp & 3, group = (warp - UNPACK_WARP0) >> 2;
        const int local_row = quadrant * 32 + lane, row = n0 + local_row;
        const bool inside = row < shape.n;
        const __half *row_scales = scales + static_cast<size_t>(inside ? row : 0) * groups;
        const __half *row_minimums = minimums + static_cast<size_t>(inside ? row : 0) * groups;
        const uint32_t code_full_u = smem_u32(code_full);
        // The loop is not unrolled: every CTA starts with a cold instruction cache, and unrolled over several steps
        // waiting for instructions was the largest stall.
        int local = group;
        uint32_t scale_next = local < steps ? load_scale_pair<PAIRED>(row_scales, 2 * (first + local), groups, inside) : 0u;
        uint32_t minimum_next = local < steps ? load_scale_pair<PAIRED>(row_minimums, 2 * (first + local), groups, inside) : 0u;
        uint32_t s = group / CODE_STEPS, phase = 0;  // the chunk of this group's step
        // A slot is free when the MMAs of the step four before are done.
        const uint32_t free_u = smem_u32(step_done);
        int before = group - A_SLOTS, before_phase = 0;
        const uint32_t tmem_base = *tmem_slot, tmem_lane = tmem_base + (TMEM_COLUMNS - A_SLOTS * A_COLUMNS) + (static_cast<uint32_t>(quadrant * 32) << 16);
#pragma unroll 1
        for (; local < steps; local += UNPACK_GROUPS) {
            const uint32_t slot = local % A_SLOTS;
            if (local >= A_SLOTS && (before += A_SLOTS) >= ring) before -= ring, before_phase ^= 1;
            const uint32_t scale = scale_next, minimum = minimum_next;
            if (local + UNPACK_GROUPS < steps) {
                scale_next = load_scale_pair<PAIRED>(row_scales, 2 * (first + local + UNPACK_GROUPS), groups, inside);
                minimum_next = load_scale_pair<PAIRED>(row_minimums, 2 * (first + local + UNPACK_GROUPS), groups, inside);
            }
            if (!mbarrier_wait_uniform(code_full_u + s * 8, phase, &g_status, STATUS_WAIT_FULL | 0x8100 | s, UNPACK_BACKOFF_NS)) { alive = false; break; }
            unpack_step(smem_c + s * CODE_BYTES + local_row * 128, (local % CODE_STEPS) * 4, local_row & 7, scale, minimum, tmem_lane + slot * A_COLUMNS, [&]() {
                if (local >= A_SLOTS && !mbarrier_wait_uniform(free_u + before * 8, before_phase, &g_status, STATUS_WAIT_EMPTY | 0x8100 | slot, UNPACK_BACKOFF_NS)) alive = false;
                tcgen05_fence_after();
            });
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbarrier_arrive(&a_ready[slot]);
                mbarrier_arrive(&code_empty[s]);
            }
            if (!alive) break;
            s += UNPACK_GROUPS / CODE_STEPS;
            if (s >= static_cast<uint32_t>(code_stages)) s -= code_stages, phase ^= 1;
        }
        if (split == 1 && bias != nullptr && inside) own_bias = __ldg(bias + row);  // on its way during the last MMAs
        // Every MMA is done, so nothing of this CTA reads or writes the stages any more.
        alive = mbarrier_wait_uniform(smem_u32(done), 0, &g_status, STATUS_WAIT_TMEM_FULL | 0x8000) && alive;
        tcgen05_fence_after();
    }
    float4 add = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // a tile that is shared: of the four outputs this thread stores
    if (split > 1) {
        const float *from = bias + n0 + lane * 4;
        if (bias != nullptr && n0 + lane * 4 < shape.n) add = make_float4(__ldg(from), __ldg(from + 1), __ldg(from + 2), __ldg(from + 3));
        cluster_sync();  // every CTA of the cluster is done with its stages
    }
    if (warp >= UNPACK_WARP0 && split == 1) {
        // The accumulator, or the sum of the two, goes from registers to y: lane = weight row, so that a warp stores 32 adjacent outputs of one
        // activation row at a time. Through shared memory, in whole rows of the tile: 1024 x 3072 x 3072 19.9 us.
        const int quadrant = warp & 3, group = (warp - UNPACK_WARP0) >> 2, n = n0 + quadrant * 32 + lane;
        const uint32_t tmem_lane = *tmem_slot + (static_cast<uint32_t>(quadrant * 32) << 16);
        const int rows = shape.m - m0 < columns ? shape.m - m0 : columns;
        for (int c = group * 16; c < columns; c += 16 * UNPACK_GROUPS) {
            uint32_t r[16];
            tmem_load_32x16(tmem_lane + c, r);
            if (issuers == 2 && steps > 1) {
                uint32_t second[16];
                tmem_load_32x16(tmem_lane + TWO_ISSUERS_COLUMNS + c, second);
                tmem_load_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(second[j]));
            } else {
                tmem_load_wait();
            }
            if (n >= shape.n) continue;
            const size_t element = static_cast<size_t>(m0 + c) * shape.ldy + n;
            if (shape.y_is_half) {
                __half *out = static_cast<__half *>(y) + element;
#pragma unroll
                for (int j = 0; j < 16; ++j, out += shape.ldy)
                    if (c + j < rows) *out = __float2half_rn(__uint_as_float(r[j]) + own_bias);
            } else {
                float *out = static_cast<float *>(y) + element;
#pragma unroll
                for (int j = 0; j < 16; ++j, out += shape.ldy)
                    if (c + j < rows) *out = __uint_as_float(r[j]) + own_bias;
            }
        }
        tcgen05_fence_before();
    } else if (warp >= UNPACK_WARP0) {
        // The accumulator, or the sum of the two (lane = weight row, column = activation row) goes to the CTA that sums that activation row, in
        // shared memory as [source CTA][row of the share][weight row]: pushed, because a load from another CTA's shared
        // memory is a round trip of a thousand cycles and a store is not.
        const int quadrant = warp & 3, group = (warp - UNPACK_WARP0) >> 2;
        const uint32_t tmem_lane = *tmem_slot + (static_cast<uint32_t>(quadrant * 32) << 16);
        const uint32_t mine = smem_u32(smem) + (rank * share * BN + quadrant * 32 + lane) * 4;
        for (int c = group * 16; c < columns; c += 16 * UNPACK_GROUPS) {
            uint32_t r[16];
            tmem_load_32x16(tmem_lane + c, r);
            int owner = c / share, row = c - owner * share;
            if (issuers == 2 && steps > 1) {
                uint32_t second[16];
                tmem_load_32x16(tmem_lane + TWO_ISSUERS_COLUMNS + c, second);
                tmem_load_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(second[j]));
            } else {
                tmem_load_wait();
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                st_cluster_f32(map_to_cta(mine + row * (BN * 4), owner), __uint_as_float(r[j]));
                if (++row == share) row = 0, ++owner;
            }
        }
        tcgen05_fence_before();
    }
    if (split > 1) cluster_sync();
    else __syncthreads();
    if (warp == MMA_WARP) {
        tcgen05_fence_after();
        tmem_dealloc(*tmem_slot, TMEM_COLUMNS);
    }
    // this CTA's share of the tile's activation rows: a warp sums and stores a row of 128 outputs at a time
    const int n = n0 + lane * 4, first_row = m0 + rank * share;
    int rows = shape.m - first_row < share ? shape.m - first_row : share;
    if (rows > columns - rank * share) rows = columns - rank * share;
    if (split > 1 && n < shape.n) {
        const float4 *sums = reinterpret_cast<const float4 *>(smem) + lane;
#pragma unroll 2
        for (int row = warp; row < rows; row += THREADS / 32) {
            float4 total = sums[row * (BN / 4)];
            for (int source = 1; source < split; ++source) {
                const float4 v = sums[(source * share + row) * (BN / 4)];
                total.x += v.x, total.y += v.y, total.z += v.z, total.w += v.w;
            }
            total.x += add.x, total.y += add.y, total.z += add.z, total.w += add.w;
            const size_t element = static_cast<size_t>(first_row + row) * shape.ldy + n;
            if (shape.y_is_half) {
                const __half2 a = __floats2half2_rn(total.x, total.y), b = __floats2half2_rn(total.z, total.w);
                *reinterpret_cast<uint2 *>(static_cast<__half *>(y) + element) =
                    make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
            } else {
                *reinterpret_cast<float4 *>(static_cast<float *>(y) + element) = total;
            }
        }
    }
    if (*reinterpret_cast<volatile uint32_t *>(&g_status) != 0) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);  // a wait gave up: let bulk copies already issued land
    }
}

}  // namespace w4a16_swap
}  // namespace qi

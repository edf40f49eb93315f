// W4A16 g64 dequant-GEMM on PAIRS of CTAs (thread-block cluster of two, tcgen05 cta_group::2):
// one 256 x 256 output tile per pair. Same operator and unpacking as w4a16_gemm.cuh
// (reference: qwen_image_cuda/cuda/gemm.cu:191-268).
//
// Chosen by qi_w4a16_gemm_tile_ex only: by shape a call takes the kernels with the operands exchanged (w4a16_swap_gemm.cuh,
// w4a16_pair_swap_gemm.cuh; 4096 x 9216 x 3072: 173 us here, 163 there), which add up K in the same order.
//
// Each CTA loads its own 128 rows of x and the packed codes of HALF of the tile's 256 weight rows,
// unpacks those 128 rows to fp16 in its own shared memory, and the leader's MMA (M = 256 across the
// pair, N = 256, K = 16) reads both halves. Compared with a 256 x 256 tile on one CTA this halves
// the unpacking work per CTA, leaves 256 TMEM columns per accumulator so that two fit (the epilogue
// of one tile overlaps the main loop of the next), and puts 74 tiles in a wave instead of 148 half
// as often full.
//
//   warp 0     TMA: own x rows (completion counted on the LEADER's barrier) and own code rows (own barrier)
//   warps 8-23 unpack own code rows, two groups of eight warps taking the K blocks in turn (measured on the block's
//              four shapes at M = 4096: 1081 -> 1127 TFLOP/s against one group; same bits); when done, arrive on the
//              LEADER's `ready` barrier
//   warp 1     leader only: 4 tcgen05.mma.cta_group::2 kind::f16 per K block; commits arrive in both CTAs
//   warps 4-7  epilogue of this CTA's 128 rows; release the accumulator on the LEADER's barrier
#pragma once
#include "ptx.cuh"
#include "w4a16_gemm.cuh"

namespace qi {
namespace w4a16_pair {

using w4a16::unpack32;
constexpr int UNPACK_GROUPS = 2;  // groups of eight unpack warps that take the K blocks in turn
constexpr int THREADS = 256 + UNPACK_GROUPS * 256;
constexpr int BK = 64;
constexpr int BM = 128, BN = 256;  // per CTA rows; pair tile is 256 x 256, each CTA unpacks 128 weight rows
constexpr int PRODUCER_WARP = 0, MMA_WARP = 1, CODE_WARP = 2, EPILOGUE_WARP0 = 4, UNPACK_WARP0 = 8, UNPACK_WARPS = 8;  // per group
constexpr int ACC_STAGES = 2;
constexpr int CODE_BLOCKS = 4, CODE_STAGES = 3;  // K blocks of codes fetched together (128 bytes of a row); chunks in flight
constexpr int A_BYTES = BM * 128, B_BYTES = (BN / 2) * 128, C_BYTES = (BN / 2) * CODE_BLOCKS * 32;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr uint32_t AHEAD_BACKOFF_NS = 100;  // pause between the polls of the roles that run ahead
constexpr int BARRIER_BYTES = 512;

template <int STAGES>
struct Tile {
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + CODE_STAGES * C_BYTES + BARRIER_BYTES + 1024;
    static_assert(SMEM_BYTES <= 232448 && SMEM_BYTES >= ONE_CTA_SMEM, "shared memory budget of one CTA; one per SM: see grid_release()");
    static_assert(STAGES >= CODE_BLOCKS, "a chunk's K blocks wrap around the stages at most once");
    static_assert((3 * STAGES + 2 * CODE_STAGES + 2 * ACC_STAGES) * 8 + 8 <= BARRIER_BYTES, "barrier block");
};

template <int STAGES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_codes,
            const __half *__restrict__ scales, const __half *__restrict__ minimums,
            const float *__restrict__ bias, void *__restrict__ y, const GemmShape shape) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smem_a = smem;
    uint8_t *smem_b = smem_a + STAGES * A_BYTES;
    uint8_t *smem_c = smem_b + STAGES * B_BYTES;
    uint64_t *code_full = reinterpret_cast<uint64_t *>(smem_c + CODE_STAGES * C_BYTES);  // own codes
    uint64_t *code_empty = code_full + CODE_STAGES;
    uint64_t *a_full = code_empty + CODE_STAGES;                                // the leader's: both CTAs' x tiles
    uint64_t *ready = a_full + STAGES;                                         // the leader's: both CTAs' unpack warps
    uint64_t *empty = ready + STAGES;
    uint64_t *tmem_full = empty + STAGES;
    uint64_t *tmem_empty = tmem_full + ACC_STAGES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + ACC_STAGES);

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t cta = cluster_ctarank();  // 0 = leader
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int tiles_m = (shape.m + (2 * BM) - 1) / (2 * BM), tiles_n = (shape.n + BN - 1) / BN;
    const int tiles = tiles_m * tiles_n, k_blocks = shape.k / BK, groups = shape.k / 64;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbarrier_init(&a_full[s], 1);
            mbarrier_init(&ready[s], 2 * UNPACK_WARPS);
            mbarrier_init(&empty[s], 1);
        }
        for (int s = 0; s < CODE_STAGES; ++s) {
            mbarrier_init(&code_full[s], 1);
            mbarrier_init(&code_empty[s], UNPACK_GROUPS * UNPACK_WARPS);
        }
        for (int a = 0; a < ACC_STAGES; ++a) {
            mbarrier_init(&tmem_full[a], 1);
            mbarrier_init(&tmem_empty[a], 2 * 4);
        }
        fence_barrier_init();
    }
    if (warp == MMA_WARP) {
        tmem_alloc_pair(tmem_slot, (ACC_STAGES * BN));
        tmem_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before anything arrives on them from the other side
    tcgen05_fence_after();
    grid_wait();
    grid_release();
    const uint32_t leader_ready = map_to_cta(smem_u32(ready), 0), leader_tmem_empty = map_to_cta(smem_u32(tmem_empty), 0);
    const uint32_t tmem_base = *tmem_slot;

    // The single-threaded roles run as converged warps with one elected lane: their addresses and descriptors live in
    // uniform registers; a diverged thread takes several times as long for the same few instructions.
    if (warp == PRODUCER_WARP) {
        if (elect_one()) prefetch_tensormap(&map_x);
        const uint32_t a_full_u = smem_u32(a_full), empty_u = smem_u32(empty), a_u = smem_u32(smem_a);
        uint32_t s = 0, phase = 1;
        bool alive = true;
        for (int tile = pair; tile < tiles && alive; tile += pairs) {
            const int m0 = (tile % tiles_m) * (2 * BM) + cta * BM;
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!mbarrier_wait_uniform(empty_u + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0x7000 | s, AHEAD_BACKOFF_NS)) { alive = false; break; }
                if (elect_one()) {
                    if (cta == 0) mbarrier_arrive_expect_tx_u32(a_full_u + s * 8, 2 * A_BYTES);  // both CTAs' x tiles
                    tma_load_2d_pair_u32(a_u + s * A_BYTES, &map_x, a_full_u + s * 8, kb * BK, m0);
                }
                __syncwarp();
                if (++s == STAGES) s = 0, phase ^= 1;
            }
        }
    } else if (warp == CODE_WARP) {
        if (elect_one()) prefetch_tensormap(&map_codes);
        const uint32_t full_u = smem_u32(code_full), empty_u = smem_u32(code_empty), c_u = smem_u32(smem_c);
        uint32_t s = 0, phase = 1;
        bool alive = true;
        for (int tile = pair; tile < tiles && alive; tile += pairs) {
            const int n0 = (tile / tiles_m) * BN + cta * (BN / 2);
            for (int kb = 0; kb < k_blocks; kb += CODE_BLOCKS) {
                if (!mbarrier_wait_uniform(empty_u + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0x7300 | s, AHEAD_BACKOFF_NS)) { alive = false; break; }
                if (elect_one()) {
                    mbarrier_arrive_expect_tx_u32(full_u + s * 8, C_BYTES);
                    tma_load_2d_u32(c_u + s * C_BYTES, &map_codes, full_u + s * 8, kb * (BK / 2), n0);
                }
                __syncwarp();
                if (++s == CODE_STAGES) s = 0, phase ^= 1;
            }
        }
    } else if (warp == MMA_WARP) {
        if (cta == 0) {
            constexpr uint32_t idesc = umma_idesc_f16_f32(2 * BM, BN);
            const uint64_t a_first = umma_desc_k_sw128(smem_u32(smem_a)), b_first = umma_desc_k_sw128(smem_u32(smem_b));
            const uint32_t a_full_u = smem_u32(a_full), ready_u = smem_u32(ready), tmem_empty_u = smem_u32(tmem_empty);
            uint32_t s = 0, phase = 0, acc = 0, acc_phase = 1;
            bool alive = true;
            for (int tile = pair; tile < tiles && alive; tile += pairs) {
                if (!mbarrier_wait_uniform(tmem_empty_u + acc * 8, acc_phase, &g_status, STATUS_WAIT_TMEM_EMPTY | 0x7000 | acc)) break;
                const uint32_t tmem_acc = tmem_base + acc * BN;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbarrier_wait_uniform2(a_full_u + s * 8, phase, ready_u + s * 8, phase, &g_status, STATUS_WAIT_READY | 0x7000 | s)) { alive = false; break; }
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint64_t a_desc = a_first + s * (A_BYTES >> 4), b_desc = b_first + s * (B_BYTES >> 4);
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk)
                            umma_f16_pair(tmem_acc, a_desc + kk * 2, b_desc + kk * 2, idesc, (kb | kk) != 0 ? 1u : 0u);
                        tcgen05_commit_pair(&empty[s]);
                        if (kb + 1 == k_blocks) tcgen05_commit_pair(&tmem_full[acc]);
                    }
                    __syncwarp();
                    if (++s == STAGES) s = 0, phase ^= 1;
                }
                if (++acc == ACC_STAGES) acc = 0, acc_phase ^= 1;
            }
        }
    } else if (warp >= UNPACK_WARP0) {
        // Eight warps unpack one K block (a thread: half a weight row, 32 codes); with more than one group of eight
        // the groups take the K blocks in turn, so that one group's waits and fences overlap the other's arithmetic.
        const int unpacker = threadIdx.x - UNPACK_WARP0 * 32;
        const int d = unpacker & 255, group = unpacker >> 8;
        const int half_row = d & 1, local_row = d >> 1;
        const uint32_t code_full_u = smem_u32(code_full), empty_u = smem_u32(empty);
        uint32_t base = 0, base_phase = 1, chunk = 0, chunk_phase = 0;  // stage of the chunk's first K block; the chunk
        bool alive = true;
        for (int tile = pair; tile < tiles && alive; tile += pairs) {
            const int row_global = (tile / tiles_m) * BN + cta * (BN / 2) + local_row;
            const bool inside = row_global < shape.n;
            const __half *row_scales = scales + static_cast<size_t>(inside ? row_global : 0) * groups;
            const __half *row_minimums = minimums + static_cast<size_t>(inside ? row_global : 0) * groups;
            const __half nothing = __ushort_as_half(0);
#pragma unroll 1
            for (int first = 0; first < k_blocks && alive; first += CODE_BLOCKS) {
                __half scale[CODE_BLOCKS / UNPACK_GROUPS], minimum[CODE_BLOCKS / UNPACK_GROUPS];
#pragma unroll
                for (int t = 0; t < CODE_BLOCKS / UNPACK_GROUPS; ++t) {
                    const int kb = first + group + t * UNPACK_GROUPS;
                    scale[t] = inside && kb < k_blocks ? __ldg(row_scales + kb) : nothing, minimum[t] = inside && kb < k_blocks ? __ldg(row_minimums + kb) : nothing;
                }
                if (!mbarrier_wait_uniform(code_full_u + chunk * 8, chunk_phase, &g_status, STATUS_WAIT_FULL | 0x7100 | chunk)) { alive = false; break; }
                const uint8_t *codes = smem_c + chunk * C_BYTES + local_row * 128;  // 16-byte pieces swizzled by the row
#pragma unroll
                for (int t = 0; t < CODE_BLOCKS / UNPACK_GROUPS; ++t) {
                    const int offset = group + t * UNPACK_GROUPS;
                    if (first + offset >= k_blocks) break;
                    const uint4 packed = *reinterpret_cast<const uint4 *>(codes + (((2 * offset + half_row) ^ (local_row & 7)) << 4));
                    uint32_t s = base + offset, phase = base_phase;
                    if (s >= STAGES) s -= STAGES, phase ^= 1;
                    uint4 out[4];
                    unpack32(packed, __half2half2(scale[t]), __half2half2(minimum[t]), out);
                    // the tensor cores are done with what the stage held before
                    if (!mbarrier_wait_uniform(empty_u + s * 8, phase, &g_status, STATUS_WAIT_EMPTY | 0x7100 | s)) { alive = false; break; }
                    uint8_t *b_row = smem_b + s * B_BYTES + local_row * 128;
#pragma unroll
                    for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4 *>(b_row + (((half_row * 4 + j) ^ (local_row & 7)) << 4)) = out[j];
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbarrier_arrive_cluster(leader_ready + s * 8);
                }
                __syncwarp();
                if (lane == 0) mbarrier_arrive(&code_empty[chunk]);
                if (++chunk == CODE_STAGES) chunk = 0, chunk_phase ^= 1;
                base += k_blocks - first < CODE_BLOCKS ? k_blocks - first : CODE_BLOCKS;
                if (base >= STAGES) base -= STAGES, base_phase ^= 1;
            }
        }
    } else if (warp >= EPILOGUE_WARP0 && warp < EPILOGUE_WARP0 + 4) {
        const int quadrant = warp & 3;  // TMEM lanes 32*quadrant .. +31 belong to this warp
        uint32_t tile_count = 0;
        for (int tile = pair; tile < tiles; tile += pairs, ++tile_count) {
            const int m0 = (tile % tiles_m) * (2 * BM) + cta * BM, n0 = (tile / tiles_m) * BN;
            const uint32_t acc = tile_count % ACC_STAGES, acc_phase = (tile_count / ACC_STAGES) & 1;
            if (!mbarrier_wait_warp(&tmem_full[acc], acc_phase, &g_status, STATUS_WAIT_TMEM_FULL | 0x7000 | acc, lane)) break;
            tcgen05_fence_after();
            {
                const int row = m0 + quadrant * 32 + lane;
                const uint32_t tmem_row = tmem_base + acc * BN + (static_cast<uint32_t>(quadrant * 32) << 16);
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    uint32_t r[32];
                    tmem_load_32x32(tmem_row + c * 32, r);
                    tmem_load_wait();
                    const int col = n0 + c * 32;
                    if (row < shape.m && col < shape.n) {
                        if (bias != nullptr) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __ldg(bias + col + j));
                        }
                        if (shape.y_is_half) {
                            __half *out = static_cast<__half *>(y) + static_cast<size_t>(row) * shape.ldy + col;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                uint32_t h[4];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const __half2 pair = __floats2half2_rn(__uint_as_float(r[8 * j + 2 * i]), __uint_as_float(r[8 * j + 2 * i + 1]));
                                    h[i] = *reinterpret_cast<const uint32_t *>(&pair);
                                }
                                reinterpret_cast<uint4 *>(out)[j] = make_uint4(h[0], h[1], h[2], h[3]);
                            }
                        } else {
                            float *out = static_cast<float *>(y) + static_cast<size_t>(row) * shape.ldy + col;
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                reinterpret_cast<uint4 *>(out)[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                        }
                    }
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbarrier_arrive_cluster(leader_tmem_empty + acc * 8);
        }
    }

    // teardown: nothing of this CTA may still be in flight when TMEM and shared memory go away
    tcgen05_fence_before();
    __syncthreads();
    if (*reinterpret_cast<volatile uint32_t *>(&g_status) != 0) {
        // a wait gave up: let bulk copies that were already issued land before the CTA exits
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    __syncwarp();
    cluster_sync();  // neither CTA may leave while the other can still reach its shared memory or barriers
    if (warp == MMA_WARP) {
        __syncwarp();
        tcgen05_fence_after();
        tmem_dealloc_pair(tmem_base, (ACC_STAGES * BN));
    }
}

}  // namespace w4a16_pair
}  // namespace qi

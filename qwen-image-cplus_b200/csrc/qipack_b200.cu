// C ABI of the library (include/qipack_b200.h): argument checks, tensor-map encoding, tile
// selection and launches. One translation unit so that every kernel shares one status word.
#include "../../include/qipack_b200.h"

#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "quantize.cuh"
#include "w4a16_gemm.cuh"
#include "w4a16_gemv.cuh"
#include "w4a16_gemv_stream.cuh"
#include "w4a16_pair_gemm.cuh"
#include "w4a16_swap_gemm.cuh"
#include "w4a16_pair_swap_gemm.cuh"
#include "w4a4_gemm.cuh"
#include "w4a4_wide_gemm.cuh"
#include "w4a4_pair_gemm.cuh"
#include "w4a4_narrow_gemm.cuh"
#include "w4a4_tall_gemm.cuh"
#include "probe.cuh"

namespace qi {
namespace {

constexpr int INVALID = static_cast<int>(cudaErrorInvalidValue);

bool aligned16(const void *pointer) { return (reinterpret_cast<uintptr_t>(pointer) & 15) == 0; }

// ---- per-device facts ------------------------------------------------------------------------

constexpr int MAX_DEVICES = 64;

int current_device() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= MAX_DEVICES) return -1;
    return device;
}

// The lazily filled tables below are atomics: two host threads that meet in a first call both do the
// (idempotent) query or cudaFuncSetAttribute, and neither reads a half-written entry.
int sm_count(int device) {
    static std::atomic<int> cached[MAX_DEVICES];
    int count = cached[device].load(std::memory_order_relaxed);
    if (count == 0) {
        if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0)
            return 148;
        cached[device].store(count, std::memory_order_relaxed);
    }
    return count;
}

// Opts a kernel into its dynamic shared memory once per device; `done` is that kernel's per-device flag.
template <typename Kernel>
cudaError_t configure_once(Kernel kernel, int smem_bytes, std::atomic<bool> &done) {
    if (done.load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (error == cudaSuccess) done.store(true, std::memory_order_release);
    return error;
}

// ---- TMA descriptors ---------------------------------------------------------------------------

typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static std::atomic<EncodeTiled> cached{nullptr};
    EncodeTiled function = cached.load(std::memory_order_acquire);
    if (function == nullptr) {
        void *entry = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess) {
            function = reinterpret_cast<EncodeTiled>(entry);
            cached.store(function, std::memory_order_release);
        }
    }
    return function;
}

// A row-major [rows, row_bytes / element] matrix seen as a 2-D tensor; box = box_inner elements
// x box_rows rows. Out-of-range rows read as zero.
bool make_map(CUtensorMap *map, CUtensorMapDataType type, int element_bytes, const void *base, uint64_t inner,
              uint64_t rows, uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_rows,
              CUtensorMapSwizzle swizzle) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows};
    const cuuint32_t element_strides[2] = {1, 1};
    (void)element_bytes;
    return encode(map, type, 2, const_cast<void *>(base), dims, strides, box, element_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- tile selection -----------------------------------------------------------------------------

// W4A16 tiles: 0 = choose by shape (never one of the others, which only qi_w4a16_gemm_tile_ex names); 1 = 128x128, 2 = 256x128,
// 3 = 128x256, 4 = 256x256, 5 = 256x256 on a pair of CTAs.

template <int NUM_M, int BN, int STAGES>
int launch_w4a16(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias,
                 void *y, const GemmShape &shape, cudaStream_t stream, int device) {
    using T = w4a16::Tile<NUM_M, BN, STAGES>;
    CUtensorMap map_x, map_codes;
    if (!make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x_half, shape.k, shape.m,
                  static_cast<uint64_t>(shape.k) * 2, 64, T::BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes, shape.k / 2, shape.n,
                  static_cast<uint64_t>(shape.k) / 2, 32, BN, CU_TENSOR_MAP_SWIZZLE_NONE))
        return INVALID;
    auto kernel = w4a16::gemm_kernel<NUM_M, BN, STAGES>;
    static std::atomic<bool> configured[MAX_DEVICES];
    if (const cudaError_t error = configure_once(kernel, T::SMEM_BYTES, configured[device])) return static_cast<int>(error);
    const int tiles = ((shape.m + T::BM - 1) / T::BM) * ((shape.n + BN - 1) / BN);
    const int grid = tiles < sm_count(device) ? tiles : sm_count(device);
    return static_cast<int>(launch_overlapped(kernel, grid, w4a16::THREADS, T::SMEM_BYTES, stream, map_x, map_codes,
                                      static_cast<const __half *>(scales), static_cast<const __half *>(minimums),
                                      bias, y, shape));
}

template <int STAGES>
int launch_w4a16_pair(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias,
                      void *y, const GemmShape &shape, cudaStream_t stream, int device) {
    namespace wp = w4a16_pair;
    using T = wp::Tile<STAGES>;
    CUtensorMap map_x, map_codes;
    if (!make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x_half, shape.k, shape.m,
                  static_cast<uint64_t>(shape.k) * 2, 64, wp::BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes, shape.k / 2, shape.n,
                  static_cast<uint64_t>(shape.k) / 2, 128, wp::BN / 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    auto kernel = wp::gemm_kernel<STAGES>;
    static std::atomic<bool> configured[MAX_DEVICES];
    if (const cudaError_t error = configure_once(kernel, T::SMEM_BYTES, configured[device])) return static_cast<int>(error);
    const int tiles = ((shape.m + 2 * wp::BM - 1) / (2 * wp::BM)) * ((shape.n + wp::BN - 1) / wp::BN);
    const int pairs = sm_count(device) / 2;
    const int grid = 2 * (tiles < pairs ? tiles : pairs);  // the kernel carries __cluster_dims__(2, 1, 1)
    return static_cast<int>(launch_overlapped(kernel, grid, wp::THREADS, T::SMEM_BYTES, stream, map_x, map_codes,
                                      static_cast<const __half *>(scales), static_cast<const __half *>(minimums),
                                      bias, y, shape));
}

// Tiles walk down the rows first, so every pass over them reads all activations again, from L2 as long as they stay there.
// Where they are larger than half of it, tiles walk through blocks of rows of which 24 MB are activations: the number of
// tiles of such a block (16384 x 9216 x 3072: 1057 -> 757 us).
int rows_in_l2(int tiles_m, long long tile_bytes) {
    if (tiles_m * tile_bytes <= (64LL << 20)) return tiles_m;
    const long long fit = (24LL << 20) / tile_bytes;
    return fit < 8 ? (tiles_m < 8 ? tiles_m : 8) : fit < tiles_m ? static_cast<int>(fit) : tiles_m;
}

// ---- the exchanged-operand kernel (w4a16_swap_gemm.cuh): its plan for a shape ----------------------------------------

template <bool PAIRED>
cudaError_t configure_swap(int device) {
    static std::atomic<bool> configured[MAX_DEVICES];
    return configure_once(w4a16_swap::gemm_kernel<PAIRED>, 232448, configured[device]);
}

void swap_config(cudaLaunchConfig_t &config, cudaLaunchAttribute (&attributes)[2], int ctas, int split, int smem_bytes, cudaStream_t stream) {
    config = {};
    config.gridDim = dim3(ctas);
    config.blockDim = dim3(w4a16_swap::THREADS);
    config.dynamicSmemBytes = smem_bytes;
    config.stream = stream;
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = split, attributes[1].val.clusterDim.y = 1, attributes[1].val.clusterDim.z = 1;
    config.attrs = attributes;
    config.numAttrs = 2;
}

// Clusters of `split` CTAs that run at the same time: fewer than SMs / split, because a cluster lies within one GPC. Asked
// of the driver once per size.
int resident_clusters(int device, int split) {
    namespace ws = w4a16_swap;
    if (split == 1) return sm_count(device);
    static std::atomic<int> cached[MAX_DEVICES][ws::MAX_SPLIT + 1];
    int count = cached[device][split].load(std::memory_order_relaxed);
    if (count == 0) {
        cudaLaunchConfig_t config;
        cudaLaunchAttribute attributes[2];
        swap_config(config, attributes, split, split, ONE_CTA_SMEM, nullptr);
        config.attrs = attributes + 1, config.numAttrs = 1;
        if (configure_swap<true>(device) != cudaSuccess || cudaOccupancyMaxActiveClusters(&count, ws::gemm_kernel<true>, &config) != cudaSuccess || count <= 0) {
            (void)cudaGetLastError();
            count = sm_count(device) / (2 * split) > 0 ? sm_count(device) / (2 * split) : 1;
        }
        cached[device][split].store(count, std::memory_order_relaxed);
    }
    return count;
}

struct SwapPlan {
    int columns, split;
    double us;  // estimated
};

// Microseconds: a step of 128 inputs costs a CTA `step` (its unpack warps) or `step_column` per column (its tensor cores and their
// operand), a tile `tile` and `tile_column` per column (its start, its first loads and its results), and sharing a tile
// over a cluster another `share` and `share_column`.
struct SwapPrices {
    double step, step_column, tile, tile_column, share, share_column;
    double us(int columns, int split, int steps, long long waves) const {
        const double a_step = columns * step_column > step ? columns * step_column : step;
        return waves * (tile + columns * tile_column + (steps + split - 1) / split * a_step + (split > 1 ? share + share_column * columns : 0.0));
    }
};
// 77 x {12288, 9216} x 3072, 16 x 18432 x 3072, {77, 256} x 3072 x 12288, {256, 1024} rows; with the weights in L2 or from HBM
constexpr SwapPrices SWAP_PRICES = {0.25, 0.003, 4.0, 0.006, 0.8, 0.016};
// Fitted to 450 shapes of 9 to 1300 rows, every width and split. They see that a narrow tile's steps cost more than the prices above
// say, and what a cluster to a wider tile then gains: 411 x 3072 x 12288 35.2 us with a CTA to 80 columns, 28.6 with two to 144.
constexpr SwapPrices SHARED_PRICES = {0.395, 0.003, 1.5, 0.0265, 1.27, 0.025};
// A cluster that is priced this much below the best tiles of one CTA takes their place: 178 such shapes of 9 to 2500 rows took 0.87 of
// the time in the mean, 0.70 to 1.01. Of 82 with prices from 1.05 to 1.1 apart three were slower, by up to 3 percent. Where the fitted
// prices chose among all tiles, 40 of 200 choices were slower by more than 2 percent: 646 x 1152 x 7616 by a third (three CTAs to a
// tile instead of two), 233 x 10528 x 576 as well (two waves instead of one), 11725 x 736 x 6848 by 9 percent (pairs).
constexpr double SHARED_GAIN = 1.1;

// Steps of 128 inputs, eight MMAs each, that are added up in one accumulator before anything is rounded to nearest. An MMA cuts its
// sum, so that the error grows with them (783 x 4096 x 12288 against 64 bits, 2-norm: 7.3e-6 with 48, 1.44e-5 with 96).
int swap_chain(int columns, int split, int steps) {
    const int issuers = w4a16_swap::issuers_of(columns), share = (steps + split - 1) / split;
    return (share + issuers - 1) / issuers;
}

// What SWAP_PRICES find best; where that is a CTA to a tile and SHARED_PRICES find it dearer by SHARED_GAIN, the cluster that they find
// best among those whose chains are no longer, so that no result is further off for it. `us` stays that of SWAP_PRICES, for the
// comparison with the pairs.
// `like`: only plans that add up K in that plan's order.
SwapPlan plan_w4a16_swap(int m, int n, int k, int device, const SwapPlan *like = nullptr) {
    namespace ws = w4a16_swap;
    const int tiles_n = (n + ws::BN - 1) / ws::BN, steps = (k + ws::BK - 1) / ws::BK;
    // The widest tiles and those a little narrower; narrower ones where all of them run at once (8192 x 32 x 64: 32 tiles of
    // 256 columns 8.2 us, 128 of 64 5.9).
    const int widest = (m + ws::MAX_COLUMNS - 1) / ws::MAX_COLUMNS;
    auto for_each = [&](auto visit) {  // columns, CTAs to a tile, waves
        for (int tiles_m = widest, before = 0; tiles_m < widest + 8 || tiles_m * tiles_n <= sm_count(device); ++tiles_m) {
            const int columns = ((m + tiles_m - 1) / tiles_m + 15) / 16 * 16;
            if (tiles_m > 1 && columns < 64) break;
            if (columns == before) continue;
            before = columns;
            if (like != nullptr && ws::issuers_of(columns) != ws::issuers_of(like->columns)) continue;
            for (int split = 1; split <= ws::MAX_SPLIT && split <= steps; ++split) {
                const long long tiles = static_cast<long long>(tiles_n) * ((m + columns - 1) / columns);
                const int resident = resident_clusters(device, split);
                const long long waves = (tiles + resident - 1) / resident;
                if (like != nullptr ? split != like->split : split > 1 && waves > 1) continue;
                visit(columns, split, waves);
            }
        }
    };
    SwapPlan best = {0, 0, 1e30};
    double dearest = 0.0;  // what a cluster may cost to take its place
    for_each([&](int columns, int split, long long waves) {
        const double us = SWAP_PRICES.us(columns, split, steps, waves);
        if (us < best.us) best = {columns, split, us}, dearest = SHARED_PRICES.us(columns, split, steps, waves) / SHARED_GAIN;
    });
    if (like != nullptr || best.split > 1) return best;
    const int chain = swap_chain(best.columns, best.split, steps);
    for_each([&](int columns, int split, long long waves) {
        const double us = SHARED_PRICES.us(columns, split, steps, waves);
        if (split > 1 && us < dearest && swap_chain(columns, split, steps) <= chain) best.columns = columns, best.split = split, dearest = us;
    });
    return best;
}

int launch_w4a16_swap(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias,
                      void *y, const GemmShape &shape, int columns, int split, cudaStream_t stream, int device) {
    namespace ws = w4a16_swap;
    CUtensorMap map_x, map_codes;
    if (!make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x_half, shape.k, shape.m,
                  static_cast<uint64_t>(shape.k) * 2, 64, columns, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes, shape.k / 2, shape.n,
                  static_cast<uint64_t>(shape.k) / 2, 128, ws::BN, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    const bool paired = ((reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(minimums)) & 3) == 0 && shape.k % 128 == 0;
    if (const cudaError_t error = paired ? configure_swap<true>(device) : configure_swap<false>(device)) return static_cast<int>(error);
    const ws::SmemPlan smem = ws::smem_plan(columns);
    const ws::Plan plan = {columns, split, smem.stages, smem.code_stages};
    const long long ctas = static_cast<long long>((shape.m + columns - 1) / columns) * ((shape.n + ws::BN - 1) / ws::BN) * split;
    if (ctas > 0x7fffffffLL) return INVALID;
    cudaLaunchConfig_t config;
    cudaLaunchAttribute attributes[2];
    swap_config(config, attributes, static_cast<int>(ctas), split, smem.bytes, stream);
    auto kernel = paired ? ws::gemm_kernel<true> : ws::gemm_kernel<false>;
    return static_cast<int>(launched(cudaLaunchKernelEx(&config, kernel, map_x, map_codes, static_cast<const __half *>(scales),
                                                        static_cast<const __half *>(minimums), bias, y, shape, plan)));
}

// The widest tile is not always the best: 4096 x 3072 outputs are 192 tiles of 256 x 256, three waves of 74 pairs, or 288 of
// 256 x 176, four waves (73.4 against 68.4 us at K = 3072). Microseconds: per column 0.0031 a step of 128 inputs and 0.0137 a
// tile (4096 x {3072, 9216, 12288} x 3072, 4096 x 3072 x 12288, 1024 x 4096 x 4096), and 3 once.
SwapPlan plan_w4a16_pair_swap(int m, int n, int k, int device) {
    namespace wp = w4a16_pair_swap;
    const int pairs = sm_count(device) / 2, steps = (k + 127) / 128;  // what fills up an even number of steps costs next to nothing
    const long long tiles_n = (n + 2 * wp::BN - 1) / (2 * wp::BN);
    SwapPlan best = {0, 2, 1e30};
    for (int columns = wp::MAX_COLUMNS; columns >= 128; columns -= 16) {
        const long long waves = (tiles_n * ((m + columns - 1) / columns) + pairs - 1) / pairs;
        const double us = 3.0 + waves * columns * (steps * 0.0031 + 0.0137);
        if (us < best.us) best = {columns, 2, us};
    }
    return best;
}

// The kernel for a shape, or for a slice of `n` of a matrix's `whole_n` weight rows. A column-sharded linear promises the bits
// of the unsharded one, and those depend on the order in which K is added up: on the number of CTAs that share it and of
// accumulators. So a slice takes the order that the whole matrix would take, and what is fastest for the slice among the
// kernels and tiles that have it. What that costs against a free choice: nothing at 4096 rows of 9216 x 3072, 8.6 against
// 7.4 us for an eighth of it at 77 rows, 19.1 against 10.3 for an eighth of 3072 x 12288 at 256.
struct W4A16Choice {
    bool pairs;  // of CTAs (w4a16_pair_swap_gemm.cuh)
    SwapPlan plan;
};
W4A16Choice choose_w4a16(int m, int n, int k, int whole_n, int device) {
    if (whole_n != n) {
        const W4A16Choice whole = choose_w4a16(m, whole_n, k, whole_n, device);
        const bool in_order = whole.pairs || (whole.plan.split == 1 && w4a16_swap::issuers_of(whole.plan.columns) == 1);  // one accumulator, all of K
        const SwapPlan pair = plan_w4a16_pair_swap(m, n, k, device);
        SwapPlan in_order_plan = {w4a16_swap::MAX_COLUMNS, 1, 0.0};
        const SwapPlan swap = plan_w4a16_swap(m, n, k, device, in_order ? &in_order_plan : &whole.plan);
        return in_order && pair.us <= swap.us ? W4A16Choice{true, pair} : W4A16Choice{false, swap};
    }
    const SwapPlan swap = plan_w4a16_swap(m, n, k, device), pair = plan_w4a16_pair_swap(m, n, k, device);
    return swap.us < pair.us ? W4A16Choice{false, swap} : W4A16Choice{true, pair};
}

int launch_w4a16_pair_swap(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias,
                           void *y, const GemmShape &shape, int columns, cudaStream_t stream, int device) {
    namespace wp = w4a16_pair_swap;
    CUtensorMap map_x, map_codes;
    if (!make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x_half, shape.k, shape.m,
                  static_cast<uint64_t>(shape.k) * 2, 64, columns / 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_codes, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes, shape.k / 2, shape.n,
                  static_cast<uint64_t>(shape.k) / 2, 128, wp::BN, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    const bool paired = ((reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(minimums)) & 3) == 0 && shape.k % 128 == 0;
    auto kernel = paired ? wp::gemm_kernel<true> : wp::gemm_kernel<false>;
    static std::atomic<bool> configured[MAX_DEVICES][2];
    if (const cudaError_t error = configure_once(kernel, wp::SMEM_BYTES, configured[device][paired])) return static_cast<int>(error);
    const int tiles = ((shape.m + columns - 1) / columns) * ((shape.n + 2 * wp::BN - 1) / (2 * wp::BN));
    const int pairs = sm_count(device) / 2;
    const int grid = 2 * (tiles < pairs ? tiles : pairs);  // the kernel carries __cluster_dims__(2, 1, 1)
    return static_cast<int>(launch_overlapped(kernel, grid, wp::THREADS, wp::SMEM_BYTES, stream, map_x, map_codes,
                                              static_cast<const __half *>(scales), static_cast<const __half *>(minimums),
                                              bias, y, shape, columns, rows_in_l2((shape.m + columns - 1) / columns, 2LL * columns * shape.k)));
}

template <int BN, int STAGES>
int launch_w4a4(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales,
                const float *bias, void *y, int32_t *dots, const GemmShape &shape, cudaStream_t stream, int device) {
    using T = w4a4::Tile<BN, STAGES>;
    CUtensorMap map_a, map_w;
    if (!make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_codes, shape.k / 2, shape.m,
                  static_cast<uint64_t>(shape.k) / 2, 64, T::BM, CU_TENSOR_MAP_SWIZZLE_NONE))
        return INVALID;
    if (!make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w_codes, shape.k / 2, shape.n,
                  static_cast<uint64_t>(shape.k) / 2, 64, BN, CU_TENSOR_MAP_SWIZZLE_NONE))
        return INVALID;
    auto kernel = dots != nullptr ? w4a4::gemm_kernel<BN, STAGES, true> : w4a4::gemm_kernel<BN, STAGES, false>;
    static std::atomic<bool> configured[MAX_DEVICES][2];
    if (const cudaError_t error = configure_once(kernel, T::SMEM_BYTES, configured[device][dots != nullptr]))
        return static_cast<int>(error);
    const int tiles = ((shape.m + T::BM - 1) / T::BM) * ((shape.n + BN - 1) / BN);
    const int grid = tiles < sm_count(device) ? tiles : sm_count(device);
    return static_cast<int>(launch_overlapped(kernel, grid, w4a4::THREADS, T::SMEM_BYTES, stream, map_a, map_w,
                                      static_cast<const __half *>(a_scales), static_cast<const __half *>(w_scales),
                                      bias, y, dots, shape));
}

template <int STAGES>
int launch_w4a4_wide(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                     const float *bias, void *y, int32_t *dots, const GemmShape &shape, cudaStream_t stream, int device) {
    using T = w4a4_wide::Tile<STAGES>;
    CUtensorMap map_a, map_w;
    if (!make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_bytes, shape.k, shape.m, static_cast<uint64_t>(shape.k),
                  w4a4_wide::STAGE_K, w4a4_wide::BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w_bytes, shape.k, shape.n, static_cast<uint64_t>(shape.k),
                  w4a4_wide::STAGE_K, w4a4_wide::BN, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    auto kernel = dots != nullptr ? w4a4_wide::gemm_kernel<STAGES, true> : w4a4_wide::gemm_kernel<STAGES, false>;
    static std::atomic<bool> configured[MAX_DEVICES][2];
    if (const cudaError_t error = configure_once(kernel, T::SMEM_BYTES, configured[device][dots != nullptr]))
        return static_cast<int>(error);
    const int tiles = ((shape.m + w4a4_wide::BM - 1) / w4a4_wide::BM) * ((shape.n + w4a4_wide::BN - 1) / w4a4_wide::BN);
    const int grid = tiles < sm_count(device) ? tiles : sm_count(device);
    return static_cast<int>(launch_overlapped(kernel, grid, w4a4_wide::THREADS, T::SMEM_BYTES, stream, map_a, map_w,
                                      static_cast<const __half *>(a_scales), static_cast<const __half *>(w_scales),
                                      bias, y, dots, shape));
}

// `peers`: the tile goes into every GPU's copy of the output. Else `dots`: y is float32 without bias, and the groups' dots are written too.
int launch_w4a4_pair(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                     const float *bias, void *y, int32_t *dots, const GemmShape &shape, cudaStream_t stream, int device,
                     const w4a4_pair::PeerOutputs *peers) {
    namespace wp = w4a4_pair;
    CUtensorMap map_a, map_w;
    if (!make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_bytes, shape.k, shape.m, static_cast<uint64_t>(shape.k),
                  128, wp::BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w_bytes, shape.k, shape.n, static_cast<uint64_t>(shape.k),
                  128, wp::B_BOX_ROWS, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if ((peers != nullptr) == (dots != nullptr)) return INVALID;
    auto kernel = peers != nullptr ? wp::gemm_kernel<true> : wp::gemm_kernel<false>;
    static std::atomic<bool> configured[MAX_DEVICES][2];
    if (const cudaError_t error = configure_once(kernel, wp::SMEM_BYTES, configured[device][peers != nullptr]))
        return static_cast<int>(error);
    const wp::PeerOutputs outputs = peers != nullptr ? *peers : wp::PeerOutputs{};
    const int pairs = sm_count(device) / 2, tiles = ((shape.m + 2 * wp::BM - 1) / (2 * wp::BM)) * ((shape.n + wp::BN - 1) / wp::BN);
    const int grid = 2 * (tiles < pairs ? tiles : pairs);  // the kernel carries __cluster_dims__(2, 1, 1)
    return static_cast<int>(launch_overlapped(kernel, grid, wp::THREADS, wp::SMEM_BYTES, stream, map_a, map_w,
                                              static_cast<const __half *>(a_scales), static_cast<const __half *>(w_scales),
                                              bias, y, dots, shape, outputs));
}

// How the tall kernel's tiles cover the output (see w4a4_tall::Tiling).
w4a4_tall::Tiling w4a4_tall_tiling(const GemmShape &shape, int ctas) {
    namespace wt = w4a4_tall;
    const int tiles_m = (shape.m + wt::BM - 1) / wt::BM, tiles_n = (shape.n + wt::BN - 1) / wt::BN, tiles = tiles_m * tiles_n;
    const int block = rows_in_l2(tiles_m, static_cast<long long>(wt::BM) * shape.k), last = (tiles_m - 1) / block * block, last_rows = tiles_m - last;
    wt::Tiling tiling = {tiles, tiles, wt::BN, tiles_m, tiles_n, block, last, last_rows, 0, 0, 0, 0};
    const int wide = tiles / ctas * ctas, before_tail = last_rows * tiles_n - (tiles - wide);  // wide tiles of the last block
    if (wide == tiles || before_tail < 0) return tiling;
    const int tail_row = before_tail % last_rows, tail_n = before_tail / last_rows * wt::BN;
    for (int width = 16; width < wt::BN; width += 16) {
        const int later = shape.n > tail_n + wt::BN ? (shape.n - tail_n - wt::BN + width - 1) / width : 0, sooner = (shape.n - tail_n + width - 1) / width;
        const int narrow = tail_row * later + (last_rows - tail_row) * sooner;
        if (narrow <= ctas) return {wide + narrow, wide, width, tiles_m, tiles_n, block, last, last_rows, tail_row, tail_n, later, sooner};
    }
    return tiling;
}

int launch_w4a4_tall(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales, const float *bias,
                     void *y, const GemmShape &shape, cudaStream_t stream, int device) {
    namespace wt = w4a4_tall;
    CUtensorMap map_a, map_w;
    if (!make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_bytes, shape.k, shape.m, static_cast<uint64_t>(shape.k),
                  wt::SLAB_K, wt::BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w_bytes, shape.k, shape.n, static_cast<uint64_t>(shape.k),
                  wt::SLAB_K, wt::BN, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    static std::atomic<bool> configured[MAX_DEVICES];
    if (const cudaError_t error = configure_once(wt::gemm_kernel, wt::SMEM_BYTES, configured[device])) return static_cast<int>(error);
    const wt::Tiling tiling = w4a4_tall_tiling(shape, sm_count(device));
    const int grid = tiling.tiles < sm_count(device) ? tiling.tiles : sm_count(device);
    return static_cast<int>(launch_overlapped(wt::gemm_kernel, grid, wt::THREADS, wt::SMEM_BYTES, stream, map_a, map_w,
                                              static_cast<const __half *>(a_scales), static_cast<const __half *>(w_scales), bias, y, shape, tiling));
}

template <int BN, bool EXCHANGED>
int launch_w4a4_narrow(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales, const float *bias,
                       void *y, const GemmShape &shape, cudaStream_t stream, int device) {
    namespace wn = w4a4_narrow;
    using T = wn::Tile<BN>;
    const int rows = EXCHANGED ? shape.n : shape.m, columns = EXCHANGED ? shape.m : shape.n;
    // rows that do not exist are not loaded: what the tensor cores make of the rest of the tile nobody reads
    const int box_rows = rows >= wn::BM ? wn::BM : (rows + 15) / 16 * 16;
    CUtensorMap map_rows, map_columns;
    if (!make_map(&map_rows, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, EXCHANGED ? w_bytes : a_bytes, shape.k, rows, static_cast<uint64_t>(shape.k),
                  128, box_rows, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    if (!make_map(&map_columns, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, EXCHANGED ? a_bytes : w_bytes, shape.k, columns, static_cast<uint64_t>(shape.k),
                  128, BN, CU_TENSOR_MAP_SWIZZLE_128B))
        return INVALID;
    static std::atomic<bool> configured[MAX_DEVICES];
    if (const cudaError_t error = configure_once(wn::gemm_kernel<BN, EXCHANGED>, T::SMEM_BYTES, configured[device])) return static_cast<int>(error);
    const int tiles = ((rows + wn::BM - 1) / wn::BM) * ((columns + BN - 1) / BN);
    const int grid = tiles < sm_count(device) ? tiles : sm_count(device);
    return static_cast<int>(launch_overlapped(wn::gemm_kernel<BN, EXCHANGED>, grid, wn::THREADS, T::SMEM_BYTES, stream, map_rows, map_columns,
                                              static_cast<const __half *>(EXCHANGED ? w_scales : a_scales),
                                              static_cast<const __half *>(EXCHANGED ? a_scales : w_scales), bias, y, shape, box_rows));
}

// Byte operands with k a multiple of 256 and 8-byte aligned scales: tall tiles (256 x 64), tiles of 128 rows by 64 or 32
// outputs, or of 128 outputs by 16, 32 or 48 activation rows; the values are the entry point's (qi_w4a4_gemm_plan).
enum W4A4Tiles { W4A4_TALL, W4A4_COLUMNS_64, W4A4_COLUMNS_32, W4A4_ROWS_16, W4A4_ROWS_32, W4A4_ROWS_48 };

// The tiles that are estimated to be fastest. A wave costs microseconds of its own and microseconds per group of 64 inputs;
// what every kernel pays once (2.6) is left out. Fitted to 677 shapes (9 to 16384 rows, 512 to 18432 outputs, 256 to 12288
// inputs, another matrix of weights every launch): within 2 to 6 % of each kernel's times, and the tiles chosen are
// 0.3 % slower than the best of the six in the mean. Prices without K, and 15 % more for every wave after the first, were 3.5 % off (264 x
// 9568 x 3328 37.9 us in tall tiles, 29.5 in 48 rows; 308 x 12288 x 3072 41.5 and 35.1; 708 x 1568 x 4096 19.8 in 128 x 32, 15.5 in tall ones).
//   far_rows: where rows lie a multiple of 4096 bytes apart their loads are slower, and the kernels that wait for loads lose
//     by it (593 x 4096 x 4096 34.6 us in 48 rows, 31.4 in tall tiles; 771 x 3072 x 3072 21.9 and 24.5), but for one tile of up to 16 rows
//   large: every tile of activation rows reads all weights, from DRAM where L2 does not hold them (190 x 8896 x 9728 47.6 us
//     in 48 rows, 42.0 in tall tiles)
W4A4Tiles choose_w4a4(const GemmShape &shape, int sms) {
    namespace wn = w4a4_narrow;
    const double groups = shape.k / 64;
    const bool far_rows = shape.k % 4096 == 0, large = static_cast<long long>(shape.n) * shape.k > (64LL << 20);
    const long long tiles_m = (shape.m + wn::BM - 1) / wn::BM, tiles_n = (shape.n + wn::BM - 1) / wn::BM;
    const auto columns_us = [&](int columns, double wave, double group) {
        return ((tiles_m * ((shape.n + columns - 1) / columns) + sms - 1) / sms) * (wave + groups * group);
    };
    const auto rows_us = [&](int rows, double wave, double group) {
        const double again = large && shape.m > rows ? 1.1 : 1.0;
        return ((tiles_n * ((shape.m + rows - 1) / rows) + sms - 1) / sms) * (wave + groups * group * again);
    };
    const w4a4_tall::Tiling tiling = w4a4_tall_tiling(shape, sms);
    const bool cut = tiling.tiles > tiling.wide;
    const int wide_waves = (tiling.wide + sms - 1) / sms;
    const double last = !cut ? 0.0 : tiling.width == 48 ? 0.207 : tiling.width == 32 ? 0.15 : 0.125;
    const struct {
        W4A4Tiles tiles;
        double us;
    } prices[] = {
        {W4A4_ROWS_16, rows_us(16, 0.75, far_rows ? 0.110 : 0.073)},
        {W4A4_ROWS_32, rows_us(32, 0.80, far_rows && shape.m > 16 ? 0.124 : 0.0957)},
        {W4A4_ROWS_48, rows_us(48, 0.93, far_rows ? 0.150 : 0.1157)},
        {W4A4_COLUMNS_64, columns_us(64, 1.30, far_rows ? 0.173 : 0.144)},
        {W4A4_COLUMNS_32, columns_us(32, 0.71, far_rows ? 0.108 : 0.090)},
        {W4A4_TALL, 0.6 + (wide_waves + cut) * 1.5 + groups * (wide_waves * 0.23 + last)},
    };
    int best = 0;
    for (int i = 1; i < 6; ++i)
        if (prices[i].us < prices[best].us) best = i;
    return prices[best].tiles;
}

// Whether the byte-operand GEMM of n outputs that comes next (n = 0: not known) takes any but tall tiles.
bool narrow_w4a4(int m, int n, int k, int sms) { return m > 0 && n > 0 && k > 0 && choose_w4a4({m, n, k, n, 0}, sms) != W4A4_TALL; }

int launch_w4a4_bytes(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales, const float *bias,
                      void *y, const GemmShape &shape, cudaStream_t stream, int device) {
    switch (choose_w4a4(shape, sm_count(device))) {
        case W4A4_ROWS_16: return launch_w4a4_narrow<16, true>(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
        case W4A4_ROWS_32: return launch_w4a4_narrow<32, true>(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
        case W4A4_ROWS_48: return launch_w4a4_narrow<48, true>(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
        case W4A4_COLUMNS_64: return launch_w4a4_narrow<64, false>(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
        case W4A4_COLUMNS_32: return launch_w4a4_narrow<32, false>(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
        default: return launch_w4a4_tall(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
    }
}

bool output_ok(const void *y, int y_dtype, long long ldy, int n) {
    if (y == nullptr || !aligned16(y) || ldy < n) return false;
    if (y_dtype == QI_DTYPE_F32) return ldy % 4 == 0;
    if (y_dtype == QI_DTYPE_F16) return ldy % 8 == 0;
    return false;
}

__global__ void dequantize_kernel(const uint8_t *__restrict__ codes, const __half *__restrict__ scales,
                                  const __half *__restrict__ minimums, __half *__restrict__ out, int n, int k) {
    // one thread per 16 code bytes (32 inputs, half a group)
    const long long chunks = static_cast<long long>(n) * (k / 32);
    const long long chunk = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (chunk >= chunks) return;
    const long long row = chunk / (k / 32);
    const int in_row = static_cast<int>(chunk % (k / 32));
    const int group = in_row / 2;
    const uint4 packed = __ldg(reinterpret_cast<const uint4 *>(codes + row * (k / 2)) + in_row);
    const __half2 scale2 = __half2half2(__ldg(scales + row * (k / 64) + group));
    const __half2 minimum2 = __half2half2(__ldg(minimums + row * (k / 64) + group));
    uint4 values[4];
    w4a16::unpack32(packed, scale2, minimum2, values);
    uint4 *destination = reinterpret_cast<uint4 *>(out + row * k + in_row * 32);
#pragma unroll
    for (int j = 0; j < 4; ++j) destination[j] = values[j];
}

// The streaming GEMV, one CTA per SM: as many stages as fit beside the activations and the partial sums. The slices of K follow
// from k alone, since the order of the sums follows from them (w4a16_gemv_stream.cuh): a row's bits must not depend on how
// many rows, or which part of a matrix, a call has. Microseconds with 3, 4 and 6 slices, one row: 18432 x 3072 9.5, 9.3, 9.5 (60 of
// them 304, 314, 322), 12288 x 4096 10.4, 10.1, 9.9 (330, 306, 281), 9216 x 2560 6.0, 5.95, 5.8 (137, 144, 148), 18432 x 1536 6.0, 6.5,
// 6.3 (194, 199, 210), 9216 x 1024 3.9, 3.7, 3.9. Two steps of K occupy half a team of four, but fewer teams disturb the copies
// less: 60 x 18432 x 512 with teams of 2, 3 and 4 139, 137, 113.
// Where a CTA has few tiles, or the stages are few, three slices are for teams of six with half of every group a warp: one and
// eight rows of 18432 x 3072 9.25 and 11.7 with teams of three, 9.3 and 11.1 with six, of 9216 x 3072 7.0 and 8.2, 6.7 and 7.8,
// of 3072 x 3072 4.7 and 6.15, 4.35 and 5.7, 60 x 18432 x 3072 297 and 332.
constexpr int STREAM_CTA_BYTES = 232448 - 1024;  // the rest is the barriers'
struct StreamPlan {
    int stages, team_warps, smem_bytes;
    bool halves;
};
StreamPlan plan_stream(int m, int k, long long tiles, int ctas) {
    const int fixed = w4a16::stream_fixed_bytes(m, k), stage = w4a16::stream_stage_bytes(k), steps = w4a16::stream_steps(k);
    int stages = (STREAM_CTA_BYTES - fixed) / stage;
    stages = stages > w4a16::STREAM_MAX_STAGES ? w4a16::STREAM_MAX_STAGES : stages;
    const int slices = steps == 1 ? 2 : steps <= 4 ? 4 : steps <= 12 ? 3 : 6;
    const bool halves = slices == 3 && (tiles < 6LL * ctas || stages < 7);
    return {stages, halves ? 2 * slices : slices, stages * stage + fixed, halves};
}

int w4a16_gemv(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias,
               void *y, int y_dtype, long long ldy, int m, int n, int k, int whole_n, cudaStream_t stream) {
    if (m < 1 || m > 8 || n <= 0 || k <= 0 || n % 16 != 0 || k % 64 != 0) return INVALID;
    if (!x_half || !codes || !scales || !minimums || !y) return INVALID;
    if (!aligned16(x_half) || !aligned16(codes) || (k % 8) != 0) return INVALID;
    if (ldy < n || (y_dtype != QI_DTYPE_F32 && y_dtype != QI_DTYPE_F16)) return INVALID;
    // Rows short enough for 16 of them to fit a stage, and regions that bulk copies can take: the streaming kernel.
    if (k <= w4a16::STREAM_MAX_K && aligned16(scales) && aligned16(minimums)) {
        const int device = current_device();
        if (device < 0) return INVALID;
        const int tiles = n / w4a16::STREAM_ROWS, resident = sm_count(device);
        const StreamPlan plan = plan_stream(m, k, tiles, resident);
        auto kernel = plan.halves ? w4a16::gemv_stream_kernel<true> : w4a16::gemv_stream_kernel<false>;
        static std::atomic<bool> configured[MAX_DEVICES][2];
        if (const cudaError_t error = configure_once(kernel, STREAM_CTA_BYTES, configured[device][plan.halves])) return static_cast<int>(error);
        if (plan.stages >= 1) {
            return static_cast<int>(launch_overlapped(kernel, tiles < resident ? tiles : resident,
                                      w4a16::STREAM_THREADS, plan.smem_bytes, stream, static_cast<const __half *>(x_half),
                                      static_cast<const uint8_t *>(codes), static_cast<const __half *>(scales),
                                      static_cast<const __half *>(minimums), bias, y, m, n, k, ldy,
                                      y_dtype == QI_DTYPE_F16, plan.stages, plan.team_warps));
        }
    }
    // Longer rows: the exchanged-operand GEMM kernel, whose clusters split K, where its alignments hold (5 x 4096 x 12288:
    // 12.2 us against 17.2 by the kernel below).
    if (n % 32 == 0 && output_ok(y, y_dtype, ldy, n)) {
        const int device = current_device();
        if (device < 0) return INVALID;
        const SwapPlan whole = plan_w4a16_swap(m, whole_n, k, device);  // see choose_w4a16
        const SwapPlan plan = whole_n == n ? whole : plan_w4a16_swap(m, n, k, device, &whole);
        const GemmShape shape = {m, n, k, ldy, y_dtype == QI_DTYPE_F16};
        return launch_w4a16_swap(x_half, codes, scales, minimums, bias, y, shape, plan.columns, plan.split, stream, device);
    }
    const int quads = (k / 64 + 3) / 4;
    int k_splits = 1;
    for (int candidate = 8; candidate >= 1; candidate /= 2)
        if (quads % candidate == 0) { k_splits = candidate; break; }
    const int row_tiles = w4a16::GEMV_WARPS / k_splits;
    const int blocks = (n / 16 + row_tiles - 1) / row_tiles;
    return static_cast<int>(launch_overlapped(w4a16::gemv_kernel, blocks, w4a16::GEMV_THREADS, 0, stream,
                                      static_cast<const __half *>(x_half), static_cast<const uint8_t *>(codes),
                                      static_cast<const __half *>(scales), static_cast<const __half *>(minimums),
                                      bias, y, m, n, k, ldy, y_dtype == QI_DTYPE_F16, k_splits));
}

// Several matrices of one shape against the same activations: launches of up to STREAM_GROUP matrices each.
int w4a16_gemv_grouped(const void *x_half, const qi_gemv_item *items, int count, int y_dtype, long long ldy, int m, int n,
                       int k, cudaStream_t stream) {
    if (m < 1 || m > 8 || n <= 0 || k <= 0 || n % 16 != 0 || k % 64 != 0 || count < 1 || items == nullptr) return INVALID;
    if (!x_half || !aligned16(x_half) || k > w4a16::STREAM_MAX_K) return INVALID;
    if (ldy < n || (y_dtype != QI_DTYPE_F32 && y_dtype != QI_DTYPE_F16)) return INVALID;
    for (int i = 0; i < count; ++i) {
        const qi_gemv_item &item = items[i];
        if (!item.codes || !item.scales || !item.minimums || !item.y) return INVALID;
        if (!aligned16(item.codes) || !aligned16(item.scales) || !aligned16(item.minimums)) return INVALID;
    }
    const int device = current_device();
    if (device < 0) return INVALID;
    const int resident = sm_count(device);
    const long long most_tiles = static_cast<long long>(count < w4a16::STREAM_GROUP ? count : w4a16::STREAM_GROUP) * (n / w4a16::STREAM_ROWS);
    const StreamPlan plan = plan_stream(m, k, most_tiles, resident);
    if (plan.stages < 1) return INVALID;
    auto kernel = plan.halves ? w4a16::gemv_stream_grouped_kernel<true> : w4a16::gemv_stream_grouped_kernel<false>;
    static std::atomic<bool> configured[MAX_DEVICES][2];
    if (const cudaError_t error = configure_once(kernel, STREAM_CTA_BYTES, configured[device][plan.halves])) return static_cast<int>(error);
    for (int first = 0; first < count; first += w4a16::STREAM_GROUP) {
        const int now = count - first < w4a16::STREAM_GROUP ? count - first : w4a16::STREAM_GROUP;
        w4a16::StreamItems group;
        for (int i = 0; i < now; ++i) {
            const qi_gemv_item &item = items[first + i];
            group.item[i] = {static_cast<const uint8_t *>(item.codes), static_cast<const __half *>(item.scales),
                             static_cast<const __half *>(item.minimums), item.bias, item.y};
        }
        for (int i = now; i < w4a16::STREAM_GROUP; ++i) group.item[i] = {nullptr, nullptr, nullptr, nullptr, nullptr};
        const long long tiles = static_cast<long long>(now) * (n / w4a16::STREAM_ROWS);
        const cudaError_t launched = launch_overlapped(kernel, tiles < resident ? static_cast<int>(tiles) : resident,
                                                       w4a16::STREAM_THREADS, plan.smem_bytes, stream, static_cast<const __half *>(x_half), group,
                                                       now, m, n, k, ldy, y_dtype == QI_DTYPE_F16, plan.stages, plan.team_warps);
        if (launched != cudaSuccess) return static_cast<int>(launched);
    }
    return 0;
}

int w4a16_gemm(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias,
               void *y, int y_dtype, long long ldy, int m, int n, int k, int whole_n, int tile, cudaStream_t stream) {
    if (m <= 0 || n <= 0 || k <= 0 || n % 32 != 0 || k % 64 != 0) return INVALID;
    if (!x_half || !codes || !scales || !minimums) return INVALID;
    if (!aligned16(x_half) || !aligned16(codes) || !output_ok(y, y_dtype, ldy, n)) return INVALID;
    const int device = current_device();
    if (device < 0) return INVALID;
    const GemmShape shape = {m, n, k, ldy, y_dtype == QI_DTYPE_F16};
    if (tile == 0) {
        // The exchanged-operand kernels: single CTAs and clusters, or persistent pairs, whichever is estimated to be faster.
        const W4A16Choice choice = choose_w4a16(m, n, k, whole_n, device);
        if (choice.pairs) return launch_w4a16_pair_swap(x_half, codes, scales, minimums, bias, y, shape, choice.plan.columns, stream, device);
        return launch_w4a16_swap(x_half, codes, scales, minimums, bias, y, shape, choice.plan.columns, choice.plan.split, stream, device);
    }
    switch (tile) {
        case 1: return launch_w4a16<1, 128, 6>(x_half, codes, scales, minimums, bias, y, shape, stream, device);
        case 2: return launch_w4a16<2, 128, 4>(x_half, codes, scales, minimums, bias, y, shape, stream, device);
        case 3: return launch_w4a16<1, 256, 4>(x_half, codes, scales, minimums, bias, y, shape, stream, device);
        case 4: return launch_w4a16<2, 256, 3>(x_half, codes, scales, minimums, bias, y, shape, stream, device);
        case 5: return launch_w4a16_pair<5>(x_half, codes, scales, minimums, bias, y, shape, stream, device);
        default: return INVALID;
    }
}

int w4a16_linear(const void *x_half, const void *codes, const void *scales, const void *minimums, const float *bias, void *y, int y_dtype,
          long long ldy, int m, int n, int k, int whole_n, cudaStream_t stream) {
    if (m >= 1 && m <= 8 && n % 16 == 0) return w4a16_gemv(x_half, codes, scales, minimums, bias, y, y_dtype, ldy, m, n, k, whole_n, stream);
    return w4a16_gemm(x_half, codes, scales, minimums, bias, y, y_dtype, ldy, m, n, k, whole_n, 0, stream);
}

// single_cta: always 128 x 128 tiles (w4a4_wide); otherwise what launch_w4a4_bytes chooses, where the shape and pointers allow.
int w4a4_gemm_wide(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                   const float *bias, void *y, int y_dtype, long long ldy, int32_t *dots, int m, int n, int k,
                   bool single_cta, cudaStream_t stream) {
    if (m <= 0 || n <= 0 || k <= 0 || n % 32 != 0 || k % 128 != 0) return INVALID;
    if (!a_bytes || !a_scales || !w_bytes || !w_scales) return INVALID;
    if (!aligned16(a_bytes) || !aligned16(w_bytes) || (reinterpret_cast<uintptr_t>(a_scales) & 3) ||
        (reinterpret_cast<uintptr_t>(w_scales) & 3) || !output_ok(y, y_dtype, ldy, n))
        return INVALID;
    const int device = current_device();
    if (device < 0) return INVALID;
    const GemmShape shape = {m, n, k, ldy, y_dtype == QI_DTYPE_F16};
    // The other kernels stage both scale arrays four groups, eight bytes, at a time; anything
    // else goes to the 128 x 128 tiles, which takes two groups per stage and four-byte-aligned scales.
    const bool scales_aligned8 = ((reinterpret_cast<uintptr_t>(a_scales) | reinterpret_cast<uintptr_t>(w_scales)) & 7) == 0;
    if (single_cta || k % w4a4_pair::STAGE_K != 0 || !scales_aligned8)
        return launch_w4a4_wide<6>(a_bytes, a_scales, w_bytes, w_scales, bias, y, dots, shape, stream, device);
    if (dots == nullptr) return launch_w4a4_bytes(a_bytes, a_scales, w_bytes, w_scales, bias, y, shape, stream, device);
    return launch_w4a4_pair(a_bytes, a_scales, w_bytes, w_scales, bias, y, dots, shape, stream, device, nullptr);
}

// The W4A4 GEMM on nibble-packed codes (the reference's operand format). `path`: 1 = the int8 kernel that widens the
// nibbles in shared memory; 2 = both operands widened to one byte per code in scratch memory (one small kernel), then
// the byte-operand kernels, which are faster by more than the widening costs once the matrices are large or the rows
// long; 0 = by shape, by the rule below. Same bits on every path. The scratch is (m + n) * k bytes from the library's own memory pool (cudaMallocFromPoolAsync) and goes
// back with cudaFreeAsync, both in stream order; if the pool refuses, path 0 falls back to 1.
constexpr int W4A4_PATHS = 3;

// The library's own memory pool for that scratch, one per device, made at first use. The device's default pool gives
// its memory back to the system at every synchronisation (release threshold 0), so a caller that synchronises
// between calls would pay a round trip to the driver per call (measured: 1.0-1.7 ms instead of 0.32 ms for the
// 4096 x 9216 x 3072 linear); this pool keeps what it has handed out until qi_w4a4_scratch_trim.
cudaMemPool_t scratch_pool(int device) {
    static std::atomic<cudaMemPool_t> pools[MAX_DEVICES];
    cudaMemPool_t pool = pools[device].load(std::memory_order_acquire);
    if (pool != nullptr) return pool;
    cudaMemPoolProps properties = {};
    properties.allocType = cudaMemAllocationTypePinned;
    properties.handleTypes = cudaMemHandleTypeNone;
    properties.location.type = cudaMemLocationTypeDevice;
    properties.location.id = device;
    if (cudaMemPoolCreate(&pool, &properties) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    unsigned long long keep = ~0ull;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPool_t expected = nullptr;
    if (!pools[device].compare_exchange_strong(expected, pool, std::memory_order_acq_rel)) {
        cudaMemPoolDestroy(pool);  // another host thread was first
        pool = expected;
    }
    return pool;
}
// One launch widens both operands: the second would add ~2 us to calls of 10.
int launch_widen_codes(const void *a_codes, void *a_bytes, long long a_rows, const void *w_codes, void *w_bytes, long long w_rows,
                       int k, cudaStream_t stream) {
    constexpr long long PER_BLOCK = w4a4_wide::WIDEN_THREADS * w4a4_wide::WIDEN_PIECES;
    const w4a4_wide::Widening a = {static_cast<const uint8_t *>(a_codes), static_cast<uint8_t *>(a_bytes), a_rows * (k / 16)};
    const w4a4_wide::Widening w = {static_cast<const uint8_t *>(w_codes), static_cast<uint8_t *>(w_bytes), w_rows * (k / 16)};
    const long long a_blocks = (a.pieces + PER_BLOCK - 1) / PER_BLOCK, w_blocks = (w.pieces + PER_BLOCK - 1) / PER_BLOCK;
    if (a_blocks + w_blocks > 0x7fffffffLL) return INVALID;
    return static_cast<int>(launch_overlapped(w4a4_wide::widen_codes_kernel, static_cast<unsigned>(a_blocks + w_blocks),
                                              w4a4_wide::WIDEN_THREADS, 0, stream, a, w, static_cast<int>(a_blocks)));
}
bool capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
        (void)cudaGetLastError();  // the legacy stream during another's capture: the launch will say so
        return false;
    }
    return status != cudaStreamCaptureStatusNone;
}

int w4a4_gemm(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales, const float *bias,
              void *y, int y_dtype, long long ldy, int32_t *dots, int m, int n, int k, int path, cudaStream_t stream) {
    if (m <= 0 || n <= 0 || k <= 0 || n % 32 != 0 || k % 128 != 0 || path < 0 || path >= W4A4_PATHS) return INVALID;
    if (!a_codes || !a_scales || !w_codes || !w_scales) return INVALID;
    if (!aligned16(a_codes) || !aligned16(w_codes) || (reinterpret_cast<uintptr_t>(a_scales) & 3) ||
        (reinterpret_cast<uintptr_t>(w_scales) & 3) || !output_ok(y, y_dtype, ldy, n))
        return INVALID;
    const int device = current_device();
    if (device < 0) return INVALID;
    const GemmShape shape = {m, n, k, ldy, y_dtype == QI_DTYPE_F16};
    const bool scales_aligned8 = ((reinterpret_cast<uintptr_t>(a_scales) | reinterpret_cast<uintptr_t>(w_scales)) & 7) == 0;
    const bool bytes_take_it = dots == nullptr && k % w4a4_pair::STAGE_K == 0 && scales_aligned8;
    if (path == 2 && !bytes_take_it) return INVALID;
    // Widening first (two launches, ~9 us at the least) against the int8 kernel, whose time is k's: 0.01 us per element
    // and tile, 9 us at k = 768 whatever m and n. Measured, int8 and widened: 1 x 128 x 3072 29.9 and 9.1 us, 77 x 9216 x
    // 3072 32.8 and 17.2, 4096 x 32 x 3072 30.8 and 11.4, 1 x 18432 x 3072 31.5 and 28.2, 1 x 32 x 256 5.9 and 9.4,
    // 255 x 4096 x 256 9.0 and 9.3; with more tiles than SMs the widened form leads at any k.
    // Not under stream capture where the int8 kernel will do: scratch makes a graph with allocation nodes, of which CUDA allows
    // one instance and no clone or child, and a caller that captures a prompt's calls may want several.
    const bool large = m >= 256 && n >= 256;
    if (path == 2 || (path == 0 && bytes_take_it && (large || (k >= 768 && !capturing(stream))))) {
        const size_t a_bytes = (static_cast<size_t>(m) * k + 255) & ~static_cast<size_t>(255);
        const size_t w_bytes = static_cast<size_t>(n) * k;
        uint8_t *scratch = nullptr;
        const cudaMemPool_t pool = scratch_pool(device);
        const cudaError_t allocated = pool == nullptr ? cudaErrorMemoryAllocation
                                                      : cudaMallocFromPoolAsync(reinterpret_cast<void **>(&scratch), a_bytes + w_bytes, pool, stream);
        if (allocated == cudaSuccess) {
            int status = launch_widen_codes(a_codes, scratch, m, w_codes, scratch + a_bytes, n, k, stream);
            if (status == 0)
                status = launch_w4a4_bytes(scratch, a_scales, scratch + a_bytes, w_scales, bias, y, shape, stream, device);
            const cudaError_t freed = cudaFreeAsync(scratch, stream);
            return status != 0 ? status : static_cast<int>(freed);
        }
        (void)cudaGetLastError();  // the refusal is not the caller's error
        if (path == 2) return static_cast<int>(allocated);
    }
    return launch_w4a4<128, 4>(a_codes, a_scales, w_codes, w_scales, bias, y, dots, shape, stream, device);
}

}  // namespace
}  // namespace qi

using namespace qi;

extern "C" {

int qi_w4a4_quantize_activations_ex(const void *x, int x_dtype, void *codes, void *scales, int m, int k, void *stream) {
    if (m < 0 || k <= 0 || k % 256 != 0) return INVALID;
    if (x_dtype != QI_DTYPE_F32 && x_dtype != QI_DTYPE_F16) return INVALID;
    if (m == 0) return 0;
    if (!x || !codes || !scales || !aligned16(x) || (reinterpret_cast<uintptr_t>(codes) & 7) ||
        (reinterpret_cast<uintptr_t>(scales) & 1))
        return INVALID;
    return static_cast<int>(launch_quantize_activations(x, x_dtype == QI_DTYPE_F16, codes, scales, nullptr, m, k,
                                                        static_cast<cudaStream_t>(stream)));
}

// next_n: outputs of the byte-operand GEMM behind it, 0 = not known.
static int quantize_wide(const void *x, int x_dtype, void *codes, void *scales, void *bytes, int m, int k, int next_n, void *stream) {
    if (m < 0 || k <= 0 || k % 256 != 0) return INVALID;
    if (x_dtype != QI_DTYPE_F32 && x_dtype != QI_DTYPE_F16) return INVALID;
    if (m == 0) return 0;
    if (!x || !scales || !bytes || !aligned16(x) || !aligned16(bytes) || (reinterpret_cast<uintptr_t>(codes) & 7) ||
        (reinterpret_cast<uintptr_t>(scales) & 1))
        return INVALID;
    return static_cast<int>(launch_quantize_activations(x, x_dtype == QI_DTYPE_F16, codes, scales, bytes, m, k,
                                                        static_cast<cudaStream_t>(stream), narrow_w4a4(m, next_n, k, quantize_sms())));
}

int qi_w4a4_quantize_activations_wide_ex(const void *x, int x_dtype, void *codes, void *scales, void *bytes, int m,
                                         int k, void *stream) {
    return quantize_wide(x, x_dtype, codes, scales, bytes, m, k, 0, stream);
}

int qi_w4a4_quantize_plan(int m, int k, int n, int sms, int *plan) {
    if (m <= 0 || k <= 0 || k % 256 != 0 || n < 0 || sms < 2 || plan == nullptr) return INVALID;
    const QuantizePlan chosen = plan_quantize(m, k, sms, narrow_w4a4(m, n, k, sms));
    plan[0] = chosen.threads;
    plan[1] = chosen.smem_bytes;
    return 0;
}

static int fused_quantize(int producer, const float *first, const float *second, void *codes, void *scales, void *bytes,
                          int m, int k, void *stream) {
    if (m < 0 || k <= 0 || k % 256 != 0) return INVALID;
    if (m == 0) return 0;
    if (!first || (producer == 1 && !second) || !scales || (!codes && !bytes)) return INVALID;
    if (!aligned16(first) || (second && !aligned16(second)) || (bytes && !aligned16(bytes)) ||
        (reinterpret_cast<uintptr_t>(codes) & 7) || (reinterpret_cast<uintptr_t>(scales) & 1))
        return INVALID;
    return static_cast<int>(launch_fused_quantize(producer, first, second, codes, scales, bytes, m, k, static_cast<cudaStream_t>(stream)));
}

int qi_w4a4_swiglu_quantize_ex(const float *gate, const float *up, void *codes, void *scales, void *bytes, int m, int k,
                               void *stream) {
    return fused_quantize(1, gate, up, codes, scales, bytes, m, k, stream);
}

int qi_w4a4_gelu_quantize_ex(const float *x, void *codes, void *scales, void *bytes, int m, int k, void *stream) {
    return fused_quantize(2, x, nullptr, codes, scales, bytes, m, k, stream);
}

int qi_w4a4_widen_codes_ex(const void *codes, void *bytes, long long rows, int k, void *stream) {
    if (rows < 0 || k <= 0 || k % 32 != 0) return INVALID;
    if (rows == 0) return 0;
    if (!codes || !bytes || !aligned16(codes) || !aligned16(bytes)) return INVALID;
    return launch_widen_codes(codes, bytes, rows, nullptr, nullptr, 0, k, static_cast<cudaStream_t>(stream));
}

int qi_w4a4_gemm_wide_ex(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                         const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, void *stream) {
    return w4a4_gemm_wide(a_bytes, a_scales, w_bytes, w_scales, bias, y, y_dtype, ldy, nullptr, m, n, k, false,
                          static_cast<cudaStream_t>(stream));
}

int qi_w4a4_gemm_plan(int m, int n, int k, int sms, int *plan) {
    if (m <= 0 || n <= 0 || k <= 0 || n % 32 != 0 || k % w4a4_pair::STAGE_K != 0 || sms < 2 || plan == nullptr) return INVALID;
    const GemmShape shape = {m, n, k, n, 0};
    const w4a4_tall::Tiling tiling = w4a4_tall_tiling(shape, sms);
    plan[0] = choose_w4a4(shape, sms);
    plan[1] = tiling.wide;
    plan[2] = tiling.tiles - tiling.wide;
    plan[3] = tiling.width;
    plan[4] = tiling.block;
    plan[5] = tiling.last_rows;
    return 0;
}

int qi_w4a4_gemm_wide_single_ex(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                                const float *bias, void *y, int y_dtype, long long ldy, int32_t *dots, int m, int n,
                                int k, void *stream) {
    return w4a4_gemm_wide(a_bytes, a_scales, w_bytes, w_scales, bias, y, y_dtype, ldy, dots, m, n, k, true,
                          static_cast<cudaStream_t>(stream));
}

int qi_w4a4_gemm_wide_scatter_ex(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                                 const float *bias, void *const *y_copies, int copies, int first_copy, int y_dtype,
                                 long long ldy, int column, int m, int n, int k, void *stream) {
    namespace wp = w4a4_pair;
    if (y_copies == nullptr || copies < 1 || copies > wp::MAX_PEERS || first_copy < 0 || first_copy >= copies)
        return INVALID;
    if (m <= 0 || n <= 0 || k <= 0 || n % 32 != 0 || k % wp::STAGE_K != 0 || column < 0 || column % 32 != 0) return INVALID;
    if (!a_bytes || !a_scales || !w_bytes || !w_scales) return INVALID;
    // this entry point always runs on CTA pairs, whose scale staging copies eight bytes at a time
    if (!aligned16(a_bytes) || !aligned16(w_bytes) || (reinterpret_cast<uintptr_t>(a_scales) & 7) ||
        (reinterpret_cast<uintptr_t>(w_scales) & 7))
        return INVALID;
    if (y_dtype != QI_DTYPE_F16 && y_dtype != QI_DTYPE_F32) return INVALID;
    if (ldy < static_cast<long long>(column) + n) return INVALID;
    const size_t element = y_dtype == QI_DTYPE_F16 ? 2 : 4;
    wp::PeerOutputs outputs = {};
    outputs.count = copies;
    outputs.first = first_copy;
    for (int i = 0; i < copies; ++i) {
        if (y_copies[i] == nullptr) return INVALID;
        outputs.y[i] = static_cast<char *>(y_copies[i]) + static_cast<size_t>(column) * element;
        if (!output_ok(outputs.y[i], y_dtype, ldy, n) || (reinterpret_cast<uintptr_t>(outputs.y[i]) & 31)) return INVALID;
    }
    if ((ldy * static_cast<long long>(element)) % 32 != 0) return INVALID;  // the epilogue stores whole 32-byte sectors
    const int device = current_device();
    if (device < 0) return INVALID;
    const GemmShape shape = {m, n, k, ldy, y_dtype == QI_DTYPE_F16};
    return launch_w4a4_pair(a_bytes, a_scales, w_bytes, w_scales, bias, outputs.y[first_copy], nullptr, shape,
                            static_cast<cudaStream_t>(stream), device, &outputs);
}

int qi_w4a4_group_dots_wide_ex(const void *a_bytes, const void *a_scales, const void *w_bytes, const void *w_scales,
                               float *y, int32_t *dots, int m, int n, int k, void *stream) {
    if (dots == nullptr) return INVALID;
    return w4a4_gemm_wide(a_bytes, a_scales, w_bytes, w_scales, nullptr, y, QI_DTYPE_F32, n, dots, m, n, k, false,
                          static_cast<cudaStream_t>(stream));
}

int qi_w4a4_quantize_activations(const float *x, void *codes, void *scales, int m, int k) {
    return qi_w4a4_quantize_activations_ex(x, QI_DTYPE_F32, codes, scales, m, k, nullptr);
}

int qi_w4a4_gemm_ex(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales,
                    const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, void *stream) {
    return w4a4_gemm(a_codes, a_scales, w_codes, w_scales, bias, y, y_dtype, ldy, nullptr, m, n, k, 0,
                     static_cast<cudaStream_t>(stream));
}

int qi_w4a4_scratch_trim(void) {
    const int device = current_device();
    if (device < 0) return INVALID;
    const cudaMemPool_t pool = scratch_pool(device);
    if (pool == nullptr) return static_cast<int>(cudaErrorMemoryAllocation);
    return static_cast<int>(cudaMemPoolTrimTo(pool, 0));
}

int qi_w4a4_gemm_path_ex(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales,
                         const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, int path, void *stream) {
    return w4a4_gemm(a_codes, a_scales, w_codes, w_scales, bias, y, y_dtype, ldy, nullptr, m, n, k, path,
                     static_cast<cudaStream_t>(stream));
}

}  // extern "C"

// ---- the packed W4A4 GEMM for callers that must not allocate ------------------------------------------------------
// The widened operands of qi_w4a4_gemm_noalloc_ex live in this array instead of pool memory. One array per device
// (the runtime gives every device its own instance of a __device__ variable), shared by every call on that device:
// calls that overlap in time - two streams, two host threads - write over each other's operands. Nothing in it has
// to start at zero: a call writes every byte it later reads, so there is nothing to clear between calls.
constexpr size_t NOALLOC_SCRATCH_BYTES = static_cast<size_t>(QI_NOALLOC_SCRATCH_BYTES);
static __device__ __align__(256) uint8_t g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

extern "C" {

int qi_w4a4_gemm_noalloc_ex(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales,
                            const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, void *stream) {
    if (m <= 0 || n <= 0 || k <= 0 || n % 32 != 0 || k % w4a4_pair::STAGE_K != 0) return INVALID;
    if (!a_codes || !a_scales || !w_codes || !w_scales) return INVALID;
    if (!aligned16(a_codes) || !aligned16(w_codes) || !output_ok(y, y_dtype, ldy, n)) return INVALID;
    if (((reinterpret_cast<uintptr_t>(a_scales) | reinterpret_cast<uintptr_t>(w_scales)) & 7) != 0) return INVALID;
    const size_t a_bytes = (static_cast<size_t>(m) * k + 255) & ~static_cast<size_t>(255);
    const size_t w_bytes = static_cast<size_t>(n) * k;
    if (a_bytes + w_bytes > NOALLOC_SCRATCH_BYTES) return QI_NOALLOC_TOO_LARGE;
    const int device = current_device();
    if (device < 0) return INVALID;
    // Set-up, once per device, with that device current: where this device's instance of the array is. It happens in
    // the first call on the device, which may also be what makes the runtime load this library's device code; make
    // that call before any stream capture begins.
    static std::atomic<uint8_t *> address[MAX_DEVICES];
    uint8_t *scratch = address[device].load(std::memory_order_acquire);
    if (scratch == nullptr) {
        const cudaError_t found = cudaGetSymbolAddress(reinterpret_cast<void **>(&scratch), g_noalloc_scratch);
        if (found != cudaSuccess) return static_cast<int>(found);
        if (scratch == nullptr) return INVALID;
        address[device].store(scratch, std::memory_order_release);
    }
    const cudaStream_t on = static_cast<cudaStream_t>(stream);
    const int status = launch_widen_codes(a_codes, scratch, m, w_codes, scratch + a_bytes, n, k, on);
    if (status != 0) return status;
    const GemmShape shape = {m, n, k, ldy, y_dtype == QI_DTYPE_F16};
    return launch_w4a4_bytes(scratch, a_scales, scratch + a_bytes, w_scales, bias, y, shape, on, device);
}

int qi_w4a4_gemm(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales, float *y,
                 int m, int n, int k) {
    if (m % 128 != 0 || n % 128 != 0 || k % 256 != 0) return INVALID;  // gemm.cu:185
    return w4a4_gemm(a_codes, a_scales, w_codes, w_scales, nullptr, y, QI_DTYPE_F32, n, nullptr, m, n, k, 0, nullptr);
}

int qi_w4a4_group_dots_ex(const void *a_codes, const void *a_scales, const void *w_codes, const void *w_scales,
                          float *y, int32_t *dots, int m, int n, int k, void *stream) {
    if (dots == nullptr) return INVALID;
    return w4a4_gemm(a_codes, a_scales, w_codes, w_scales, nullptr, y, QI_DTYPE_F32, n, dots, m, n, k, 1,
                     static_cast<cudaStream_t>(stream));
}

int qi_w4a16_gemv_ex(const void *x_half, const void *codes, const void *scales, const void *minimums,
                     const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, void *stream) {
    return w4a16_gemv(x_half, codes, scales, minimums, bias, y, y_dtype, ldy, m, n, k, n, static_cast<cudaStream_t>(stream));
}

int qi_w4a16_gemv_grouped_ex(const void *x_half, const qi_gemv_item *items, int count, int y_dtype, long long ldy, int m,
                             int n, int k, void *stream) {
    return w4a16_gemv_grouped(x_half, items, count, y_dtype, ldy, m, n, k, static_cast<cudaStream_t>(stream));
}

int qi_w4a16_gemm_ex(const void *x_half, const void *codes, const void *scales, const void *minimums,
                     const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, void *stream) {
    return w4a16_linear(x_half, codes, scales, minimums, bias, y, y_dtype, ldy, m, n, k, n, static_cast<cudaStream_t>(stream));
}

int qi_w4a16_gemm_tile_ex(const void *x_half, const void *codes, const void *scales, const void *minimums,
                          const float *bias, void *y, int y_dtype, long long ldy, int m, int n, int k, int tile,
                          void *stream) {
    if (tile < 0 || tile > 5) return INVALID;
    return w4a16_gemm(x_half, codes, scales, minimums, bias, y, y_dtype, ldy, m, n, k, n, tile, static_cast<cudaStream_t>(stream));
}

int qi_w4a16_gemm(const void *x_half, const void *codes, const void *scales, const void *minimums, float *y, int m,
                  int n, int k) {
    if (m % 128 != 0 || n % 128 != 0 || k % 64 != 0) return INVALID;  // gemm.cu:264
    return w4a16_gemm(x_half, codes, scales, minimums, nullptr, y, QI_DTYPE_F32, n, m, n, k, n, 0, nullptr);
}

int qi_f32_to_f16(const float *source, void *out, unsigned long long count) {
    if (count == 0) return 0;
    if (!source || !out) return INVALID;
    return static_cast<int>(launch_f32_to_f16(source, out, count, nullptr));
}

int qi_f32_to_f16_ex(const float *source, void *out, unsigned long long count, void *stream) {
    if (count == 0) return 0;
    if (!source || !out) return INVALID;
    return static_cast<int>(launch_f32_to_f16(source, out, count, static_cast<cudaStream_t>(stream)));
}

int qi_w4a16_dequantize_ex(const void *codes, const void *scales, const void *minimums, void *w_half, int n, int k,
                           void *stream) {
    if (n <= 0 || k <= 0 || k % 64 != 0) return INVALID;
    if (!codes || !scales || !minimums || !w_half || !aligned16(codes) || !aligned16(w_half)) return INVALID;
    const long long chunks = static_cast<long long>(n) * (k / 32);
    const long long blocks = (chunks + 255) / 256;
    if (blocks > 0x7fffffffLL) return INVALID;
    dequantize_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t *>(codes), static_cast<const __half *>(scales), static_cast<const __half *>(minimums),
        static_cast<__half *>(w_half), n, k);
    return static_cast<int>(cudaGetLastError());
}

// The dispatcher for a record that holds record->n of a matrix's whole_n weight rows.
static int linear_slice(const qi_packed_linear *record, int whole_n, const qi_linear_work *work, const void *input, int input_dtype,
                        void *output, int output_dtype, long long ld_output, int rows, int reuse_input, void *stream) {
    if (!record || !work || !input || !output || rows <= 0) return INVALID;
    if (record->group_size != 64) return INVALID;
    if (input_dtype != QI_DTYPE_F32 && input_dtype != QI_DTYPE_F16) return INVALID;
    const int n = record->n, k = record->k;
    if (record->scheme == QI_SCHEME_W4A4_H256) {  // transformer.cplus:702-708
        if (!work->code_scales) return INVALID;
        if (record->weights_wide != nullptr && work->wide != nullptr) {
            // one byte per code on both sides: no unpacking inside the GEMM
            if (!reuse_input) {
                const int status = quantize_wide(input, input_dtype, work->codes, work->code_scales, work->wide, rows, k, n, stream);
                if (status != 0) return status;
            }
            return qi_w4a4_gemm_wide_ex(work->wide, work->code_scales, record->weights_wide, record->scales, record->bias,
                                        output, output_dtype, ld_output, rows, n, k, stream);
        }
        if (!work->codes) return INVALID;
        if (!reuse_input) {
            const int status = qi_w4a4_quantize_activations_ex(input, input_dtype, work->codes, work->code_scales, rows, k, stream);
            if (status != 0) return status;
        }
        return qi_w4a4_gemm_ex(work->codes, work->code_scales, record->weights, record->scales, record->bias, output,
                               output_dtype, ld_output, rows, n, k, stream);
    }
    if (record->scheme == QI_SCHEME_W4A16) {  // transformer.cplus:709-712
        const void *x_half = input;
        if (input_dtype == QI_DTYPE_F32) {
            if (!work->halves) return INVALID;
            if (!reuse_input) {
                const int status = static_cast<int>(launch_f32_to_f16(static_cast<const float *>(input), work->halves,
                                                                      static_cast<unsigned long long>(rows) * k,
                                                                      static_cast<cudaStream_t>(stream)));
                if (status != 0) return status;
            }
            x_half = work->halves;
        }
        return w4a16_linear(x_half, record->weights, record->scales, record->zeros, record->bias, output, output_dtype, ld_output, rows, n, k,
                     whole_n, static_cast<cudaStream_t>(stream));
    }
    return INVALID;
}

int qi_linear(const qi_packed_linear *record, const qi_linear_work *work, const void *input, int input_dtype,
              void *output, int output_dtype, long long ld_output, int rows, int reuse_input, void *stream) {
    return record == nullptr ? INVALID : linear_slice(record, record->n, work, input, input_dtype, output, output_dtype, ld_output, rows, reuse_input, stream);
}

int qi_kernel_status(unsigned int *status) {
    if (!status) return INVALID;
    cudaError_t error = cudaDeviceSynchronize();
    if (error != cudaSuccess) return static_cast<int>(error);
    uint32_t value = 0;
    error = cudaMemcpyFromSymbol(&value, g_status, sizeof(value));
    if (error != cudaSuccess) return static_cast<int>(error);
    if (value != 0) {
        const uint32_t zero = 0;
        error = cudaMemcpyToSymbol(g_status, &zero, sizeof(zero));
    }
    *status = value;
    return static_cast<int>(error);
}

int qi_probe_tensor_rate(int kind, double seconds, double *tera_ops_per_second) {
    if (kind < 0 || kind > 2 || !(seconds > 0.0) || seconds > 2.0 || !tera_ops_per_second) return INVALID;
    const int device = current_device();
    if (device < 0) return INVALID;
    void (*kernel)(int) = kind == 0 ? probe::mma_rate_kernel<0> : kind == 1 ? probe::mma_rate_kernel<1> : probe::mma_rate_kernel<2>;
    cudaError_t error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, probe::SMEM_BYTES);
    if (error != cudaSuccess) return static_cast<int>(error);
    const int sms = sm_count(device);
    const double ops_per_batch = 2.0 * 128 * 256 * (kind == 0 ? 16 : 32) * probe::BATCH * sms;
    cudaEvent_t begin, end;
    if ((error = cudaEventCreate(&begin)) != cudaSuccess) return static_cast<int>(error);
    if ((error = cudaEventCreate(&end)) != cudaSuccess) { cudaEventDestroy(begin); return static_cast<int>(error); }
    // a short launch sizes the long one: the rate under the power limit differs from the rate of a burst
    int batches = 64;
    float ms = 0.0f;
    for (int round = 0; round < 2 && error == cudaSuccess; ++round) {
        cudaEventRecord(begin, nullptr);
        kernel<<<sms, probe::THREADS, probe::SMEM_BYTES>>>(batches);
        cudaEventRecord(end, nullptr);
        error = cudaEventSynchronize(end);
        if (error == cudaSuccess) error = cudaEventElapsedTime(&ms, begin, end);
        if (round == 0 && error == cudaSuccess && ms > 0.0f) {
            const double wanted = seconds * 1e3 / ms * batches;
            batches = wanted > 4e6 ? 4000000 : (wanted < 64 ? 64 : static_cast<int>(wanted));
        }
    }
    cudaEventDestroy(begin);
    cudaEventDestroy(end);
    if (error != cudaSuccess) return static_cast<int>(error);
    *tera_ops_per_second = ops_per_batch * batches / (ms * 1e-3) / 1e12;
    return 0;
}

int qi_probe_wait_timeout(unsigned long long limit_ns, void *stream) {
    if (limit_ns == 0 || limit_ns > 100000000ull) return INVALID;  // at most a tenth of a second
    probe::wait_timeout_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(limit_ns);
    return static_cast<int>(cudaGetLastError());
}

const char *qi_b200_version(void) { return "qipack_b200 0.1 sm_100a"; }

}  // extern "C"

#include "shard.cuh"
#include "pack_file.cuh"

"""Parity of the CUDA kernels with the CPU oracle, through the C ABI, on a B200.

Bars (from the operator's definition): activation codes and scales, unpacked weights and
per-group integer dots bit-exact; fp32 outputs within 1e-3 of max|y|; fp16 stores within
2 fp16 ulp of the fp32 oracle rounded to fp16."""
import ctypes
import pathlib
import re

import numpy as np
import pytest

import __graft_entry__ as entry
from oracle import qipack_oracle as qo
from tests import qi_testing as qt

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OUTPUT_TOLERANCE = 1e-3  # max |y - oracle| / max |oracle|, fp32 accumulate
FP16_STORE_ULPS = 2
CSRC = pathlib.Path(entry.__file__).parent / "qwen-image-cplus_b200" / "csrc"


@pytest.fixture(scope="module")
def qi():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    module = entry.load_package()
    module.lib()  # fails loudly if the CUDA library is missing: there is no fallback
    torch.cuda.set_device(0)
    return module


def up(array):
    return torch.from_numpy(np.ascontiguousarray(array)).cuda()


def half_bits(tensor):
    return tensor.cpu().numpy().view(np.uint16)


def check_status(qi):
    torch.cuda.synchronize()
    assert qi.kernel_status() == 0


# ---- activation quantiser -------------------------------------------------------------------

@pytest.mark.parametrize("m,k", [(1, 256), (3, 512), (77, 768), (128, 3072), (517, 1024), (256, 12288)])
@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_quantize_activations_bit_exact(qi, m, k, dtype):
    rng = np.random.default_rng(1000 + m + k)
    x16 = qt.make_activations(rng, m, k)
    x = x16 if dtype == "f16" else (x16.astype(np.float32) + rng.standard_normal((m, k), dtype=np.float32) * 1e-3)
    codes = torch.zeros(m, k // 2, dtype=torch.uint8, device="cuda")
    scales = torch.zeros(m, k // 64, dtype=torch.float16, device="cuda")
    xd = up(x)
    if dtype == "f32":
        assert qi.w4a4_quantize_activations(xd, codes, scales, m, k) == 0
    else:
        assert qi.w4a4_quantize_activations_ex(xd, qi.DTYPE_F16, codes, scales, m, k) == 0
    check_status(qi)
    expected_codes, expected_scales = qo.quantize_activations(x)
    assert np.array_equal(half_bits(scales), expected_scales)
    assert np.array_equal(codes.cpu().numpy(), expected_codes)


def test_quantize_activations_rounding_ties(qi):
    # values that sit exactly on, and one fp32 step either side of, every rounding tie
    # (n + 0.5) * scale, so that the reciprocal shortcut must defer to the exact division
    rng = np.random.default_rng(77)
    m, k = 64, 1024
    # rotating H256(v) gives v back: build the wanted post-rotation values and rotate them
    target = np.zeros((m, k), dtype=np.float32)
    for row in range(m):
        for g in range(k // 64):
            scale = np.float16(rng.uniform(0.01, 2.0))
            peak = np.float32(scale) * np.float32(7.0)
            ties = (rng.integers(-7, 7, size=64).astype(np.float32) + np.float32(0.5)) * np.float32(scale)
            nudge = rng.integers(-2, 3, size=64)
            values = ties.copy()
            for _ in range(2):
                values = np.where(nudge > 0, np.nextafter(values, np.float32(np.inf)), values)
                values = np.where(nudge < 0, np.nextafter(values, np.float32(-np.inf)), values)
                nudge = nudge - np.sign(nudge)
            values[0] = peak
            target[row, g * 64:(g + 1) * 64] = values
    x = qo.hadamard_256(target)
    codes = torch.zeros(m, k // 2, dtype=torch.uint8, device="cuda")
    scales = torch.zeros(m, k // 64, dtype=torch.float16, device="cuda")
    assert qi.w4a4_quantize_activations(up(x), codes, scales, m, k) == 0
    check_status(qi)
    expected_codes, expected_scales = qo.quantize_activations(x)
    assert np.array_equal(half_bits(scales), expected_scales)
    assert np.array_equal(codes.cpu().numpy(), expected_codes)


def test_quantize_activations_zero_and_tiny_rows(qi):
    m, k = 8, 512
    x = np.zeros((m, k), dtype=np.float32)
    x[1, :] = 1e-9
    x[2, 5] = 1e-7
    x[3, :] = -3e-8
    x[4, 0::2] = 65504.0
    codes = torch.full((m, k // 2), 0xAB, dtype=torch.uint8, device="cuda")
    scales = torch.zeros(m, k // 64, dtype=torch.float16, device="cuda")
    assert qi.w4a4_quantize_activations(up(x), codes, scales, m, k) == 0
    check_status(qi)
    expected_codes, expected_scales = qo.quantize_activations(x)
    assert np.array_equal(half_bits(scales), expected_scales)
    assert np.array_equal(codes.cpu().numpy(), expected_codes)
    assert np.all(expected_scales[0] == 1)  # the 2^-24 floor (gemm.cu:45)


@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_quantize_activations_in_each_form(qi, dtype):
    # one chunk or two a half-warp, CTAs of one, two and eight warps, by the number of chunks: the bytes of the oracle, and of rows
    # with ties, infinities, NaNs, denormals and the largest values those that any other form gives
    k = 1024
    rng = np.random.default_rng(41)
    most = 8300  # chunks: 33200, past the last that one chunk a half-warp takes
    x = qt.make_activations(rng, most, k)
    x = x if dtype == "f16" else x.astype(np.float32) + rng.standard_normal((most, k), dtype=np.float32) * 1e-3
    expected_codes, expected_scales = qo.quantize_activations(x)
    special = [(0, 5, np.inf), (1, 300, -np.inf), (2, 700, np.nan), (3, slice(None), 6.1e-5), (4, slice(0, 256), 65504.0), (5, slice(None), 0.0), (6, slice(0, None, 64), 3.5), (7, 1000, np.inf), (7, 1001, -np.inf)]
    strange = x.copy()
    for row, columns, value in special:
        strange[row, columns] = value
    if dtype == "f32":
        strange[8, ::3] = 1e-40
        strange[9, ::5] = 1e30
    first = None
    for m in (10, 295, 296, 297, 767, 768, 769, 1791, 1792, 8192, 8193, most):
        for source, plain in ((x, True), (strange, False)):
            codes = torch.zeros(m, k // 2, dtype=torch.uint8, device="cuda")
            scales = torch.zeros(m, k // 64, dtype=torch.float16, device="cuda")
            wide = torch.zeros(m, k, dtype=torch.uint8, device="cuda")
            code = qi.DTYPE_F32 if dtype == "f32" else qi.DTYPE_F16
            assert qi.w4a4_quantize_activations_wide_ex(up(source[:m]), code, codes, scales, wide, m, k) == 0
            check_status(qi)
            if plain:
                assert np.array_equal(half_bits(scales), expected_scales[:m])
                assert np.array_equal(codes.cpu().numpy(), expected_codes[:m])
                nibbles = torch.zeros_like(wide)
                assert qi.w4a4_widen_codes_ex(codes, nibbles, m, k) == 0
                assert torch.equal(wide, nibbles)
            else:
                now = [t[:10].cpu().numpy().copy() for t in (codes, scales.view(torch.int16), wide)]
                first = now if first is None else first
                assert all(np.array_equal(a, b) for a, b in zip(first, now)), m


@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_quantize_activations_at_the_limits_of_its_forms(qi, dtype):
    # the last chunk count of a form and the first of the next (148 SMs), in rows of one chunk
    rng = np.random.default_rng(43)
    limits = [limit * 148 for limit in (8, 21, 48, 222)]
    x = qt.make_activations(rng, limits[-1] + 1, 256)
    x = x if dtype == "f16" else x.astype(np.float32)
    expected_codes, expected_scales = qo.quantize_activations(x)
    source = up(x)
    for m in (edge for limit in limits for edge in (limit, limit + 1)):
        codes, scales = torch.zeros(m, 128, dtype=torch.uint8, device="cuda"), torch.zeros(m, 4, dtype=torch.float16, device="cuda")
        assert qi.w4a4_quantize_activations_ex(source, qi.DTYPE_F32 if dtype == "f32" else qi.DTYPE_F16, codes, scales, m, 256) == 0
        check_status(qi)
        assert np.array_equal(half_bits(scales), expected_scales[:m])
        assert np.array_equal(codes.cpu().numpy(), expected_codes[:m])


@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_quantize_activations_in_ctas_of_four_warps(qi, dtype):
    # the first and the last row count that long rows have it for (148 SMs), one beyond either, and CTAs whose last warps have no chunk
    rng = np.random.default_rng(47)
    for k, rows in ((4352, (121, 122, 182, 183)), (12288, (44, 47, 64))):
        assert {qi.w4a4_quantize_plan(m, k).threads for m in rows[1:3]} == {128}
        x = qt.make_activations(rng, rows[-1], k)
        x = x if dtype == "f16" else x.astype(np.float32)
        expected_codes, expected_scales = qo.quantize_activations(x)
        source = up(x)
        for m in rows:
            codes, scales = torch.zeros(m, k // 2, dtype=torch.uint8, device="cuda"), torch.zeros(m, k // 64, dtype=torch.float16, device="cuda")
            wide, nibbles = torch.zeros(m, k, dtype=torch.uint8, device="cuda"), torch.zeros(m, k, dtype=torch.uint8, device="cuda")
            assert qi.w4a4_quantize_activations_wide_ex(source, qi.DTYPE_F32 if dtype == "f32" else qi.DTYPE_F16, codes, scales, wide, m, k) == 0
            check_status(qi)
            assert np.array_equal(half_bits(scales), expected_scales[:m])
            assert np.array_equal(codes.cpu().numpy(), expected_codes[:m])
            assert qi.w4a4_widen_codes_ex(codes, nibbles, m, k) == 0
            assert torch.equal(wide, nibbles)


def test_quantize_rejects_bad_shapes(qi):
    x = torch.zeros(4, 320, device="cuda")
    out = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_quantize_activations(x, out, out, 4, 320) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a4_quantize_activations(x, out, out, 0, 256) == 0  # empty input: nothing to do
    assert qi.w4a4_quantize_activations(None, out, out, 4, 256) == qi.CUDA_ERROR_INVALID_VALUE


def test_f32_to_f16_bit_exact(qi):
    rng = np.random.default_rng(3)
    for count in (1, 7, 8, 4099, 1 << 20):
        x = np.concatenate([rng.standard_normal(count).astype(np.float32) * np.float32(10.0 ** rng.integers(-8, 5)),
                            ])[:count]
        out = torch.zeros(count, dtype=torch.float16, device="cuda")
        assert qi.f32_to_f16(up(x), out, count) == 0
        torch.cuda.synchronize()
        assert np.array_equal(half_bits(out), qo.f32_to_f16(x))
        on_stream = torch.zeros(count, dtype=torch.float16, device="cuda")
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        assert qi.f32_to_f16_ex(up(x), on_stream, count, stream.cuda_stream) == 0
        stream.synchronize()
        assert np.array_equal(half_bits(on_stream), qo.f32_to_f16(x))


# ---- W4A16 ---------------------------------------------------------------------------------------

def test_w4a16_dequantize_bit_exact(qi):
    rng = np.random.default_rng(11)
    n, k = 384, 1024
    for source in ("packer", "packer_clip", "random", "wide"):
        if source.startswith("packer"):
            codes, scales, minimums = qt.pack_w4a16(qt.make_weights(rng, n, k), clip=source.endswith("clip"))
        elif source == "random":
            codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
        else:  # |w| up to 1: the edge of the range where a single rounding equals the reference's two
            codes = rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)
            scales = rng.uniform(0.01, 0.12, size=(n, k // 64)).astype(np.float16).view(np.uint16)
            minimums = rng.uniform(-0.95, -0.85, size=(n, k // 64)).astype(np.float16).view(np.uint16)
        out = torch.zeros(n, k, dtype=torch.float16, device="cuda")
        assert qi.w4a16_dequantize_ex(up(codes), up(scales), up(minimums), out, n, k) == 0
        torch.cuda.synchronize()
        expected = qo.w4a16_dequantize(codes, scales, minimums)
        assert np.abs(expected.astype(np.float32)).max() <= 1.0
        assert np.array_equal(half_bits(out), expected.view(np.uint16)), source


@pytest.mark.parametrize("tile", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 256, 512), (384, 640, 1024), (128, 384, 3072)])
def test_w4a16_gemm_matches_oracle(qi, tile, m, n, k):
    rng = np.random.default_rng(2000 + m + n + k)
    codes, scales, minimums = qt.pack_w4a16(qt.make_weights(rng, n, k))
    x16 = qt.make_activations(rng, m, k)
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemm_tile_ex(up(x16), up(codes), up(scales), up(minimums), None, y, qi.DTYPE_F32, n, m, n, k,
                                 tile) == 0
    check_status(qi)
    expected = qo.w4a16_gemm(x16, codes, scales, minimums)
    assert qt.max_relative_error(y.cpu().numpy(), expected) <= OUTPUT_TOLERANCE


def test_w4a16_gemm_default_tiles_large(qi):
    # the block shapes' to_q linear at 512x512 image size: m=1024, n=k=3072, checked on sampled rows
    rng = np.random.default_rng(31)
    m, n, k = 1024, 3072, 3072
    codes, scales, minimums = qt.pack_w4a16(qt.make_weights(rng, n, k))
    x16 = qt.make_activations(rng, m, k)
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemm(up(x16), up(codes), up(scales), up(minimums), y, m, n, k) == 0
    check_status(qi)
    got = y.cpu().numpy()
    assert np.isfinite(got).all()
    rows = np.sort(rng.choice(m, size=48, replace=False))
    expected = qo.w4a16_gemm(x16[rows], codes, scales, minimums)
    assert qt.max_relative_error(got[rows], expected) <= OUTPUT_TOLERANCE


def test_w4a16_gemm_ex_bias_fp16_and_leading_dimension(qi):
    rng = np.random.default_rng(41)
    m, n, k, ldy = 200, 256, 512, 512  # m is not a multiple of 128: the _ex form takes any m > 8
    codes, scales, minimums = qt.pack_w4a16(qt.make_weights(rng, n, k))
    x16, bias = qt.make_activations(rng, m, k), qt.make_bias(rng, n)
    expected = qo.w4a16_gemm(x16, codes, scales, minimums, bias=bias)
    wide = torch.full((m, ldy), -7.0, dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemm_ex(up(x16), up(codes), up(scales), up(minimums), up(bias), wide[:, 128:], qi.DTYPE_F32, ldy,
                            m, n, k) == 0
    check_status(qi)
    got = wide.cpu().numpy()
    assert qt.max_relative_error(got[:, 128:128 + n], expected) <= OUTPUT_TOLERANCE
    assert np.all(got[:, :128] == -7.0) and np.all(got[:, 128 + n:] == -7.0)  # nothing outside the slice
    y16 = torch.zeros(m, n, dtype=torch.float16, device="cuda")
    assert qi.w4a16_gemm_ex(up(x16), up(codes), up(scales), up(minimums), up(bias), y16, qi.DTYPE_F16, n, m, n, k) == 0
    check_status(qi)
    distance, checked = qt.fp16_store_error(y16.cpu().numpy(), expected)
    assert distance <= FP16_STORE_ULPS and checked > 0.5
    assert qt.max_relative_error(y16.cpu().numpy().astype(np.float32), expected) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("m,n,k", [(9, 32, 64), (16, 160, 192), (17, 4096, 64), (77, 288, 1216), (100, 1024, 3072), (255, 416, 448),
                                   (257, 96, 1024), (130, 3072, 128), (1, 256, 12288), (8, 480, 4160), (520, 64, 640)])
def test_w4a16_exchanged_operands_at_the_edges_of_their_tiles(qi, m, n, k):
    # rows and columns that end inside a tile, an odd number of groups, K split over a cluster and not; few enough rows
    # (or long enough ones) that the kernel with the weights as first operand takes the shape
    rng = np.random.default_rng(4000 + m + n + k)
    codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
    x16, bias = qt.make_activations(rng, m, k), qt.make_bias(rng, n)
    expected = qo.w4a16_gemm(x16, codes, scales, minimums, bias=bias)
    for dtype, code in ((torch.float32, qi.DTYPE_F32), (torch.float16, qi.DTYPE_F16)):
        wide = torch.full((m + 1, n + 32), -7.0, dtype=dtype, device="cuda")
        assert qi.w4a16_gemm_ex(up(x16), up(codes), up(scales), up(minimums), up(bias), wide, code, n + 32, m, n, k) == 0
        check_status(qi)
        got = wide.float().cpu().numpy()
        assert np.all(got[m:] == -7.0) and np.all(got[:, n:] == -7.0)  # nothing outside the matrix
        assert qt.max_relative_error(got[:m, :n], expected) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("m,n,k", [(2048, 2048, 128), (4000, 1504, 192), (3000, 2336, 1216), (9000, 288, 320),
                                   (3000, 9216, 64), (3000, 2336, 320), (2000, 4128, 640), (4096, 1504, 1088),
                                   (4096, 3072, 1024), (3300, 1504, 12288)])
def test_w4a16_exchanged_operands_on_pairs_over_several_tiles(qi, m, n, k):
    # more 256-row tiles than pairs of CTAs, ragged on both sides, an odd number of groups or of steps (one step past the
    # end of K), scales read in pairs (K a multiple of 128) and one by one, and more activations than stay in L2, walked in
    # blocks of eight rows of tiles of which the last is shorter; against the unpacked weights in float64, every output
    rng = np.random.default_rng(5000 + m + n + k)
    codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
    x, bias = up(qt.make_activations(rng, m, k)), up(qt.make_bias(rng, n))
    c, s, z = up(codes), up(scales.view(np.float16)), up(minimums.view(np.float16))
    weights = torch.empty(n, k, dtype=torch.float16, device="cuda")
    assert qi.w4a16_dequantize_ex(c, s, z, weights, n, k) == 0
    expected = (x.double() @ weights.double().T + bias.double()).cpu().numpy()
    for dtype, code in ((torch.float32, qi.DTYPE_F32), (torch.float16, qi.DTYPE_F16)):
        wide = torch.full((m + 1, n + 32), -7.0, dtype=dtype, device="cuda")
        assert qi.w4a16_gemm_ex(x, c, s, z, bias, wide, code, n + 32, m, n, k) == 0
        check_status(qi)
        got = wide.float().cpu().numpy()
        assert np.all(got[m:] == -7.0) and np.all(got[:, n:] == -7.0)  # nothing outside the matrix
        assert qt.max_relative_error(got[:m, :n], expected) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("m,n,k", [(9, 96, 3072), (77, 12288, 3072), (96, 1024, 6144), (100, 3072, 3072), (200, 9216, 3072), (256, 3072, 12288),
                                   (384, 1024, 6144), (512, 1536, 12288), (1024, 384, 3072), (1500, 1152, 3072), (300, 1024, 192)])
def test_w4a16_same_bits_on_every_call(qi, m, n, k):
    # one accumulator and two, from eight stages of activations down to three, K split over a cluster and not: the order of
    # the sums is fixed, whatever else runs at the time; and each result is the product of the unpacked weights
    rng = np.random.default_rng(5500 + m + n + k)
    codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
    x, c, s, z = up(qt.make_activations(rng, m, k)), up(codes), up(scales.view(np.float16)), up(minimums.view(np.float16))
    weights = torch.empty(n, k, dtype=torch.float16, device="cuda")
    assert qi.w4a16_dequantize_ex(c, s, z, weights, n, k) == 0
    results = [torch.full((m, n), float("nan"), device="cuda") for _ in range(8)]
    for y in results:
        assert qi.w4a16_gemm_ex(x, c, s, z, None, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert all(torch.equal(results[0], y) for y in results[1:])
    exact = x.double() @ weights.double().T
    assert float((results[0] - exact).norm() / exact.norm()) <= 1e-4  # 12288 float32 additions: 12288 ** 0.5 * 2 ** -23 = 1.3e-5


@pytest.mark.parametrize("m,n,k,steps", [(495, 7456, 5568, 22), (201, 10304, 9920, 39), (783, 4096, 12288, 48)])
def test_w4a16_gemm_sums_are_as_exact_as_short_chains(qi, m, n, k, steps):
    # as for the GEMV below: 2^-25 for each MMA of a chain, eight a step of 128 inputs, and 2^-23 for the sums of the chains. These
    # shapes have tiles of 80 to 112 columns, whose two accumulators take the steps in turn; wider ones have one and all steps in it
    rng = np.random.default_rng(3015 + m + n + k)
    codes = rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)
    scales = (rng.uniform(0.9, 1.1, size=(n, k // 64)) * 0.0065).astype(np.float16)
    minimums = (-7.5 * scales.astype(np.float32)).astype(np.float16)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(1)).half().cuda()
    nibbles = torch.stack([up(codes) & 15, up(codes) >> 4], -1).reshape(n, k // 64, 64).half().double()
    weights = (nibbles * up(scales).double()[..., None] + up(minimums).double()[..., None]).half().double().reshape(n, k)
    exact = x.double() @ weights.T
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemm_ex(x, up(codes), up(scales.view(np.uint16)), up(minimums.view(np.uint16)), None, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert float((y.double() - exact).norm() / exact.norm()) <= steps * 8 * 2.0 ** -25 + 2.0 ** -23


def test_w4a16_unpack_scales_about_its_limit(qi):
    # the unpack's fast path takes |scale| < 1/32: both sides of it, either sign, and the smallest scales there are
    n, k = 64, 1024
    rng = np.random.default_rng(3010)
    codes = rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)
    edge = np.float16(1 / 32)
    values = np.array([edge, np.nextafter(edge, np.float16(0)), np.nextafter(edge, np.float16(1)), 1 / 16, 3 / 64, 2.0 ** -24, 2.0 ** -14, 0.0065], dtype=np.float16)
    scales = (values[rng.integers(0, len(values), size=(n, k // 64))] * rng.choice([-1.0, 1.0], size=(n, k // 64))).astype(np.float16)
    minimums = rng.uniform(-0.06, 0.06, size=scales.shape).astype(np.float16)
    nibbles = np.stack([codes & 15, codes >> 4], axis=-1).reshape(n, k // 64, 64).astype(np.float64)
    expected = (nibbles * scales.astype(np.float64)[:, :, None] + minimums.astype(np.float64)[:, :, None]).astype(np.float16).reshape(n, k)  # one rounding
    weights = torch.zeros(n, k, dtype=torch.float16, device="cuda")
    assert qi.w4a16_dequantize_ex(up(codes), up(scales.view(np.uint16)), up(minimums.view(np.uint16)), weights, n, k) == 0
    check_status(qi)
    assert np.array_equal(weights.cpu().numpy().view(np.uint16), expected.view(np.uint16))


def test_w4a16_unpack_of_a_few_larger_scales_costs_little(qi):
    # a warp that has one scale of 1/32 or more among its 32 rows takes the longer unpack once, not both one after the other:
    # 13 instructions for 11, with both it would be 24 (5 % and 41 % of this call)
    m, n, k = 77, 12288, 3072
    rng = np.random.default_rng(3020)
    x, y = up(qt.make_activations(rng, m, k)), torch.zeros(m, n, dtype=torch.float16, device="cuda")
    codes = up(rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8))
    small = rng.uniform(0.006, 0.007, size=(n, k // 64)).astype(np.float16)
    mixed = np.where(rng.random(small.shape) < 0.1, np.float16(0.046), small)
    best = []
    for scales in (small, mixed):
        minimums = up((-7.5 * scales.astype(np.float32)).astype(np.float16).view(np.uint16))
        device = up(scales.view(np.uint16))
        times = []
        for _ in range(9):  # the best of them: others may use the machine
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(100):
                assert qi.w4a16_gemm_ex(x, codes, device, minimums, None, y, qi.DTYPE_F16, n, m, n, k) == 0
            end.record()
            check_status(qi)
            times.append(begin.elapsed_time(end))
        best.append(min(times))
    assert best[1] <= 1.2 * best[0], best


def test_w4a16_gemm_rejects_what_the_reference_rejects(qi):  # gemm.cu:264
    t = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    assert qi.w4a16_gemm(t, t, t, t, t, 100, 128, 64) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a16_gemm(t, t, t, t, t, 128, 120, 64) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a16_gemm(t, t, t, t, t, 128, 128, 96) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a16_gemm(None, t, t, t, t, 128, 128, 64) == qi.CUDA_ERROR_INVALID_VALUE


@pytest.mark.parametrize("m", [1, 2, 8])
@pytest.mark.parametrize("n,k,kind", [(256, 64, "silu"), (1024, 1216, "silu"), (18432, 3072, "silu"),
                                      (3072, 12288, "outliers")])
def test_w4a16_gemv_matches_oracle(qi, m, n, k, kind):
    rng = np.random.default_rng(3000 + m + n + k)
    if n * k > (1 << 22):
        codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
    else:
        codes, scales, minimums = qt.pack_w4a16(qt.make_weights(rng, n, k))
    x16, bias = qt.make_activations(rng, m, k, kind), qt.make_bias(rng, n)
    expected = qo.w4a16_gemm(x16, codes, scales, minimums, bias=bias)
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(up(x16), up(codes), up(scales), up(minimums), up(bias), y, qi.DTYPE_F32, n, m, n, k) == 0
    torch.cuda.synchronize()
    assert qt.max_relative_error(y.cpu().numpy(), expected) <= OUTPUT_TOLERANCE
    y16 = torch.zeros(m, n, dtype=torch.float16, device="cuda")
    assert qi.w4a16_gemm_ex(up(x16), up(codes), up(scales), up(minimums), up(bias), y16, qi.DTYPE_F16, n, m, n, k) == 0
    torch.cuda.synchronize()
    distance, _ = qt.fp16_store_error(y16.cpu().numpy(), expected)
    assert distance <= FP16_STORE_ULPS


@pytest.mark.parametrize("m,n,k", [(1, 48, 192), (2, 32, 512), (4, 2400, 1024), (5, 2400, 1088), (1, 21328, 1536), (3, 4784, 2880), (4, 64, 4096)])
def test_w4a16_gemv_teams_and_steps(qi, m, n, k):
    # 2, 4, 3 and 6 slices of K, last steps of one to four groups, activation rows that fill the MMA's columns to half and one more
    rng = np.random.default_rng(3050 + m + n + k)
    codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
    x16, bias = qt.make_activations(rng, m, k, "silu"), qt.make_bias(rng, n)
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(up(x16), up(codes), up(scales), up(minimums), up(bias), y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert qt.max_relative_error(y.cpu().numpy(), qo.w4a16_gemm(x16, codes, scales, minimums, bias=bias)) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("m", [1, 2, 8])
@pytest.mark.parametrize("n,k,chain", [(576, 256, 8), (2400, 512, 8), (9216, 1024, 8), (18432, 1536, 16), (6144, 2048, 24), (3072, 3072, 32), (4096, 4096, 32)])
def test_w4a16_gemv_sums_are_as_exact_as_short_chains(qi, m, n, k, chain):
    # An MMA cuts its float32 sum towards zero, on the mean by half a unit of 2^-24 to 2^-23 of it: 2^-25 for each of a chain of
    # them that only grows, plus what rounding the chains' sums to nearest adds (2^-23)
    rng = np.random.default_rng(3060 + m + n + k)
    codes = rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)
    scales = (rng.uniform(0.9, 1.1, size=(n, k // 64)) * 0.0065).astype(np.float16)
    minimums = (-7.5 * scales.astype(np.float32)).astype(np.float16)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(1)).half().cuda()
    nibbles = torch.stack([up(codes) & 15, up(codes) >> 4], -1).reshape(n, k // 64, 64).double()
    weights = (nibbles * up(scales).double()[..., None] + up(minimums).double()[..., None]).half().double().reshape(n, k)
    exact = x.double() @ weights.T
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(x, up(codes), up(scales.view(np.uint16)), up(minimums.view(np.uint16)), None, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert float((y.double() - exact).norm() / exact.norm()) <= chain * 2.0 ** -25 + 2.0 ** -23


@pytest.mark.parametrize("n,k", [(48, 64), (576, 256), (4784, 512), (2400, 704), (4784, 1024), (2400, 1088), (14224, 1536), (4784, 1984), (2400, 2048),
                                 (4784, 2560), (14224, 3072), (2400, 3136), (4784, 4096)])
def test_w4a16_gemv_rows_do_not_depend_on_their_number(qi, n, k):
    # every kind of teams, with the lower rows' codes where the others end and further on: the bits of a row of activations alone
    # are those it has among others, and against a few weight rows those against all (many are for teams of three warps, few
    # for teams of six with the same slices of K)
    rng = np.random.default_rng(3070 + n + k)
    codes, scales, minimums = (up(a) for a in qt.random_w4a16_pack(rng, n, k))
    x, bias = up(qt.make_activations(rng, 8, k, "silu")), up(qt.make_bias(rng, n))
    results = []
    for m in range(1, 9):
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        assert qi.w4a16_gemv_ex(x, codes, scales, minimums, bias, y, qi.DTYPE_F32, n, m, n, k) == 0
        results.append(y)
    check_status(qi)
    for m, y in enumerate(results, 1):
        assert torch.equal(y, results[-1][:m]), m
    alone = torch.full((1, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(x[5:], codes, scales, minimums, bias, alone, qi.DTYPE_F32, n, 1, n, k) == 0
    check_status(qi)
    assert torch.equal(alone[0], results[-1][5])
    few = torch.full((8, 48), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(x, codes[:48], scales[:48], minimums[:48], bias[:48], few, qi.DTYPE_F32, 48, 8, 48, k) == 0
    check_status(qi)
    assert torch.equal(few, results[-1][:, :48])


@pytest.mark.parametrize("m", [1, 3])
def test_w4a16_gemv_scales_of_every_size(qi, m):
    # scales from fp16 denormals up to 4: the GEMV's unpack treats scale >= 1/16 (where scale * 2^20 leaves fp16)
    # and denormal scales on paths of their own; every one must give the reference's weights
    n, k = 512, 1024
    rng = np.random.default_rng(3100 + m)
    codes = rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)
    exponents = rng.integers(-20, 3, size=(n, k // 64)).astype(np.float32)
    scales = (np.exp2(exponents) * rng.uniform(1.0, 2.0, size=exponents.shape)).astype(np.float16)
    scales[::7, ::3] = np.float16(0.0)
    minimums = (-7.5 * scales.astype(np.float32)).astype(np.float16)
    x16 = qt.make_activations(rng, m, k, "silu")
    expected = qo.w4a16_gemm(x16, codes, scales.view(np.uint16), minimums.view(np.uint16))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(up(x16), up(codes), up(scales.view(np.uint16)), up(minimums.view(np.uint16)), None, y,
                            qi.DTYPE_F32, n, m, n, k) == 0
    torch.cuda.synchronize()
    assert qt.max_relative_error(y.cpu().numpy(), expected) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("low,high", [(2.0 ** -9, 1 / 64 - 2.0 ** -16), (1 / 64, 1 / 4 - 2.0 ** -12), (1 / 4, 1.0)])
@pytest.mark.parametrize("m,n,k", [(1, 16, 64), (8, 48, 4096), (5, 2384, 1216)])
def test_w4a16_gemv_scales_of_one_range(qi, m, n, k, low, high):
    # all scales of a matrix in one of the three ranges that the unpack tells apart, both ends of each included
    rng = np.random.default_rng(3150 + m + n + k)
    codes = rng.integers(0, 256, size=(n, k // 2), dtype=np.uint8)
    scales = rng.uniform(low, high, size=(n, k // 64)).astype(np.float16)
    scales[0, 0], scales[-1, -1] = np.float16(low), np.float16(-high)
    minimums = (-7.5 * scales.astype(np.float32)).astype(np.float16)
    x16 = qt.make_activations(rng, m, k)
    expected = qo.w4a16_gemm(x16, codes, scales.view(np.uint16), minimums.view(np.uint16))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a16_gemv_ex(up(x16), up(codes), up(scales.view(np.uint16)), up(minimums.view(np.uint16)), None, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert qt.max_relative_error(y.cpu().numpy(), expected) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("m", [1, 8])
@pytest.mark.parametrize("n,k,scale_offset,output_offset", [(48, 4160, 0, 0), (16, 12288, 0, 0), (80, 3072, 1, 0), (96, 4160, 0, 1), (64, 12288, 1, 3), (48, 64, 1, 1)])
def test_w4a16_gemv_without_what_the_other_kernels_need(qi, m, n, k, scale_offset, output_offset):
    # long rows of which there is no multiple of 32, or an output that starts or steps off 16 bytes; scales off 16 bytes with
    # rows the streaming kernel would take: the kernel that reads weights and scales from global memory one by one
    rng = np.random.default_rng(3170 + m + n + k)
    codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
    x16, bias = qt.make_activations(rng, m, k), qt.make_bias(rng, n)
    expected = qo.w4a16_gemm(x16, codes, scales, minimums, bias=bias)
    shifted = []
    for values in (scales, minimums):
        room = torch.zeros(n * (k // 64) + 8, dtype=torch.float16, device="cuda")
        shifted.append(room[scale_offset:scale_offset + n * (k // 64)].copy_(up(values.view(np.float16)).flatten()))
    ldy = n + output_offset
    for dtype, code in ((torch.float32, qi.DTYPE_F32), (torch.float16, qi.DTYPE_F16)):
        room = torch.full((output_offset + (m + 1) * ldy,), -7.0, dtype=dtype, device="cuda")
        y = room[output_offset:].view(m + 1, ldy)
        assert qi.w4a16_gemv_ex(up(x16), up(codes), *shifted, up(bias), y, code, ldy, m, n, k) == 0
        check_status(qi)
        got = y.float().cpu().numpy()
        assert np.all(got[m:] == -7.0) and np.all(got[:, n:] == -7.0)
        assert qt.max_relative_error(got[:m, :n], expected) <= OUTPUT_TOLERANCE


@pytest.mark.parametrize("m,count,n,k", [(1, 3, 1024, 1216), (1, 70, 256, 512), (2, 5, 18432, 3072)])
def test_w4a16_gemv_grouped_matches_oracle_and_the_single_launches(qi, m, count, n, k):
    """Several matrices of one shape against the same activations in one launch (two for more than 64 matrices): every
    output equals the oracle's within the tolerance and the single-matrix GEMV's bit for bit."""
    rng = np.random.default_rng(3200 + m + count + n + k)
    x16 = qt.make_activations(rng, m, k, "silu")
    x = up(x16)
    entries, singles, expected = [], [], []
    for index in range(count):
        codes, scales, minimums = qt.random_w4a16_pack(rng, n, k)
        bias = qt.make_bias(rng, n) if index % 2 == 0 else None
        device = (up(codes), up(scales), up(minimums), up(bias) if bias is not None else None,
                  torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda"))
        entries.append(device)
        single = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        assert qi.w4a16_gemv_ex(x, device[0], device[1], device[2], device[3], single, qi.DTYPE_F32, n, m, n, k) == 0
        singles.append(single)
        if index < 4 or index == count - 1:  # the oracle on a few of them; the single launches cover the rest
            expected.append((index, qo.w4a16_gemm(x16, codes, scales, minimums, bias=bias)))
    table, keep = qi.gemv_items(entries)
    assert qi.w4a16_gemv_grouped_ex(x, table, qi.DTYPE_F32, n, m, n, k) == 0
    torch.cuda.synchronize()
    check_status(qi)
    for index, (entry, single) in enumerate(zip(entries, singles)):
        assert torch.equal(entry[4], single), index
    for index, want in expected:
        assert qt.max_relative_error(entries[index][4].cpu().numpy(), want) <= OUTPUT_TOLERANCE
    # refused: no items, a misaligned region, rows too long for the streaming kernel
    assert qi.lib().qi_w4a16_gemv_grouped_ex(qi._p(x), table, 0, qi.DTYPE_F32, n, m, n, k, None) == qi.CUDA_ERROR_INVALID_VALUE
    bad, _ = qi.gemv_items([(entries[0][0].view(-1)[1:], entries[0][1], entries[0][2], None, entries[0][4])])
    assert qi.w4a16_gemv_grouped_ex(x, bad, qi.DTYPE_F32, n, m, n, k) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a16_gemv_grouped_ex(x, table, qi.DTYPE_F32, n, m, n, 8192) == qi.CUDA_ERROR_INVALID_VALUE


@pytest.mark.parametrize("m,k", [(1, 256), (3, 512), (1, 1024), (1, 1088), (1, 3072), (2, 3072), (8, 3072), (1, 4096), (8, 4096)])
def test_w4a16_gemv_rings_go_round(qi, m, k):
    # each kind of teams with tiles for every stage of a CTA's ring twice and more, where the number of stages is a multiple of
    # the teams' number and where it is not: stages are handed back, fetched into again and waited for in either phase
    n, count = 1200, 64
    most_stages = int(re.search(r"STREAM_MAX_STAGES = (\d+)", (CSRC / "w4a16_gemv_stream.cuh").read_text()).group(1))
    assert count * (n // 16) > 2 * most_stages * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(3250 + m + k)
    codes, scales, minimums = qt.random_w4a16_pack(rng, count * n, k)
    x16, bias = qt.make_activations(rng, m, k, "silu"), qt.make_bias(rng, count * n)
    x, device = up(x16), [up(a) for a in (codes, scales, minimums, bias)]
    y = torch.full((count, m, n), float("nan"), dtype=torch.float32, device="cuda")
    items = [tuple(a[i * n:(i + 1) * n] for a in device) + (y[i],) for i in range(count)]
    table, keep = qi.gemv_items(items)
    assert qi.w4a16_gemv_grouped_ex(x, table, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    for i, item in enumerate(items):  # 75 tiles alone: no stage is used twice
        single = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        assert qi.w4a16_gemv_ex(x, *item[:4], single, qi.DTYPE_F32, n, m, n, k) == 0
        assert torch.equal(y[i], single), i
    check_status(qi)
    for i in (0, count // 2, count - 1):
        of = slice(i * n, (i + 1) * n)
        assert qt.max_relative_error(y[i].cpu().numpy(), qo.w4a16_gemm(x16, codes[of], scales[of], minimums[of], bias=bias[of])) <= OUTPUT_TOLERANCE


# ---- W4A4 ----------------------------------------------------------------------------------------

@pytest.mark.parametrize("m,n,k", [(128, 128, 256), (256, 384, 512), (128, 256, 3072), (384, 128, 1280)])
def test_w4a4_gemm_matches_oracle_and_dots_are_exact(qi, m, n, k):
    rng = np.random.default_rng(4000 + m + n + k)
    w_codes, w_scales = qt.pack_w4a4(qt.make_weights(rng, n, k))
    a_codes, a_scales = qo.quantize_activations(qt.make_activations(rng, m, k))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    args = (up(a_codes), up(a_scales), up(w_codes), up(w_scales))
    assert qi.w4a4_gemm(*args, y, m, n, k) == 0
    check_status(qi)
    expected = qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales)
    got = y.cpu().numpy()
    assert qt.max_relative_error(got, expected) <= OUTPUT_TOLERANCE
    # same fused multiply-adds in the same order as the reference kernel: expect the very bits
    assert np.array_equal(got, expected)
    dots = torch.full((m, n, k // 64), 12345, dtype=torch.int32, device="cuda")
    y2 = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    assert qi.w4a4_group_dots_ex(*args, y2, dots, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(dots.cpu().numpy(), qo.w4a4_group_dots(a_codes, w_codes))
    assert np.array_equal(y2.cpu().numpy(), got)


def test_w4a4_gemm_extreme_codes_and_scales(qi):
    # every code at +-7 (largest |dot| = 64*49) and scales from the 2^-24 floor to large
    m, n, k = 128, 128, 512
    a_codes = np.full((m, k // 2), 0x77, dtype=np.uint8)
    a_codes[1::2] = 0x99
    w_codes = np.full((n, k // 2), 0x77, dtype=np.uint8)
    w_codes[2::3] = 0x99
    w_codes[5::7] = 0x97
    rng = np.random.default_rng(9)
    a_scales = rng.choice(np.array([2.0 ** -24, 1e-3, 0.5, 30.0], dtype=np.float16), size=(m, k // 64)).view(np.uint16)
    w_scales = rng.choice(np.array([2.0 ** -24, 1e-4, 0.01, 2.0], dtype=np.float16), size=(n, k // 64)).view(np.uint16)
    y = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    dots = torch.zeros(m, n, k // 64, dtype=torch.int32, device="cuda")
    assert qi.w4a4_group_dots_ex(up(a_codes), up(a_scales), up(w_codes), up(w_scales), y, dots, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(dots.cpu().numpy(), qo.w4a4_group_dots(a_codes, w_codes))
    assert np.array_equal(y.cpu().numpy(), qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales))


def test_w4a4_gemm_ex_bias_fp16_and_leading_dimension(qi):
    rng = np.random.default_rng(51)
    m, n, k, ldy = 256, 256, 768, 384
    w_codes, w_scales = qt.pack_w4a4(qt.make_weights(rng, n, k))
    a_codes, a_scales = qo.quantize_activations(qt.make_activations(rng, m, k, "gelu"))
    bias = qt.make_bias(rng, n)
    expected = qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales, bias=bias)
    args = (up(a_codes), up(a_scales), up(w_codes), up(w_scales), up(bias))
    wide = torch.full((m, ldy), 3.0, dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm_ex(*args, wide, qi.DTYPE_F32, ldy, m, n, k) == 0
    check_status(qi)
    got = wide.cpu().numpy()
    assert qt.max_relative_error(got[:, :n], expected) <= OUTPUT_TOLERANCE
    assert np.all(got[:, n:] == 3.0)
    y16 = torch.zeros(m, n, dtype=torch.float16, device="cuda")
    assert qi.w4a4_gemm_ex(*args, y16, qi.DTYPE_F16, n, m, n, k) == 0
    check_status(qi)
    distance, checked = qt.fp16_store_error(y16.cpu().numpy(), expected)
    assert distance <= FP16_STORE_ULPS and checked > 0.5


def test_w4a4_gemm_block_shape_sampled(qi):
    # attention-out shape of the 1024x1024 block (m=4096, n=k=3072): full-size run, sampled rows
    rng = np.random.default_rng(61)
    m, n, k = 4096, 3072, 3072
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm(up(a_codes), up(a_scales), up(w_codes), up(w_scales), y, m, n, k) == 0
    check_status(qi)
    got = y.cpu().numpy()
    assert np.isfinite(got).all()
    rows = np.sort(rng.choice(m, size=32, replace=False))
    expected = qo.w4a4_gemm(a_codes[rows], a_scales[rows], w_codes, w_scales)
    assert np.array_equal(got[rows], expected)


@pytest.mark.parametrize("m,n,k", [(256, 384, 512), (512, 256, 3072), (200, 256, 768), (256, 256, 640)])
def test_w4a4_gemm_paths_give_the_same_bits(qi, m, n, k):
    """The packed-operand entry point on each of its kernels: the int8 kernel on nibbles, and both operands widened
    into scratch memory for the byte-operand kernels (twice in a row: the scratch is taken and returned
    in stream order)."""
    rng = np.random.default_rng(4500 + m + n + k)
    if k % 256 == 0:
        w_codes, w_scales = qt.pack_w4a4(qt.make_weights(rng, n, k))
        a_codes, a_scales = qo.quantize_activations(qt.make_activations(rng, m, k))
    else:  # not a length the H256 format has, but one the int8 kernel takes (two groups per stage)
        w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
        a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    bias = qt.make_bias(rng, n)
    expected = qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales, bias=bias)
    args = (up(a_codes), up(a_scales), up(w_codes), up(w_scales), up(bias))
    paths = [qi.W4A4_PATH_INT8, qi.W4A4_PATH_BY_SHAPE] + ([qi.W4A4_PATH_WIDENED] * 2 if k % 256 == 0 else [])
    for path in paths:
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        assert qi.w4a4_gemm_path_ex(*args, y, qi.DTYPE_F32, n, m, n, k, path) == 0
        check_status(qi)
        assert np.array_equal(y.cpu().numpy(), expected), path
    torch.cuda.synchronize()
    assert qi.w4a4_scratch_trim() == 0  # the pool gives back what no call holds; the next call takes it again
    y = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm_path_ex(*args, y, qi.DTYPE_F32, n, m, n, k, qi.W4A4_PATH_BY_SHAPE) == 0
    check_status(qi)
    assert np.array_equal(y.cpu().numpy(), expected)
    assert qi.w4a4_gemm_path_ex(*args, y, qi.DTYPE_F32, n, m, n, k, 3) == qi.CUDA_ERROR_INVALID_VALUE
    if k % 256 != 0:  # the byte-operand kernels take groups in fours
        assert qi.w4a4_gemm_path_ex(*args, y, qi.DTYPE_F32, n, m, n, k, qi.W4A4_PATH_WIDENED) == qi.CUDA_ERROR_INVALID_VALUE


def test_w4a4_gemm_rejects_what_the_reference_rejects(qi):  # gemm.cu:185
    t = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_gemm(t, t, t, t, t, 100, 128, 256) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a4_gemm(t, t, t, t, t, 128, 100, 256) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a4_gemm(t, t, t, t, t, 128, 128, 128) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.w4a4_gemm(t, None, t, t, t, 128, 128, 256) == qi.CUDA_ERROR_INVALID_VALUE


# ---- transformer::linear ---------------------------------------------------------------------------

def test_linear_dispatches_like_the_reference(qi):
    # transformer.cplus:673-713: q, k, v share one quantised / converted input (reuse_input)
    rng = np.random.default_rng(71)
    rows, n, k = 256, 384, 768
    x32 = qt.make_activations(rng, rows, k).astype(np.float32) + np.float32(1e-4)
    xd = up(x32)
    work = qi.LinearWork(torch.zeros(rows * k // 2, dtype=torch.uint8, device="cuda"),
                         torch.zeros(rows * k // 64, dtype=torch.float16, device="cuda"),
                         torch.zeros(rows * k, dtype=torch.float16, device="cuda"))
    a_codes, a_scales = qo.quantize_activations(x32)
    x_half = qo.f32_to_f16(x32).view(np.float16)
    for scheme in (qi.SCHEME_W4A4_H256, qi.SCHEME_W4A16):
        outputs = []
        for index in range(3):
            w16 = qt.make_weights(rng, n, k)
            if scheme == qi.SCHEME_W4A4_H256:
                codes, scales = qt.pack_w4a4(w16)
                record = qi.PackedLinear(scheme, n, k, up(codes), up(scales))
                expected = qo.w4a4_gemm(a_codes, a_scales, codes, scales)
            else:
                codes, scales, minimums = qt.pack_w4a16(w16)
                record = qi.PackedLinear(scheme, n, k, up(codes), up(scales), up(minimums))
                expected = qo.w4a16_gemm(x_half, codes, scales, minimums)
            y = torch.zeros(rows, n, dtype=torch.float32, device="cuda")
            assert qi.linear(record, work, xd, y, rows, reuse_input=index > 0) == 0
            check_status(qi)
            assert qt.max_relative_error(y.cpu().numpy(), expected) <= OUTPUT_TOLERANCE
            outputs.append(y)
    bad = qi.PackedLinear(3, n, k, xd, xd)
    assert qi.linear(bad, work, xd, outputs[0], rows) == qi.CUDA_ERROR_INVALID_VALUE


# ---- W4A4 on byte-wide (E4M3) operands ---------------------------------------------------------------

def e4m3_of_codes(codes):
    """Expected output of qi_w4a4_widen_codes_ex: the FP8 E4M3 encoding of each code in -8..7."""
    magnitude = np.array([0x00, 0x38, 0x40, 0x44, 0x48, 0x4A, 0x4C, 0x4E, 0x50], dtype=np.uint8)
    values = qo.unpack_codes(codes, True).astype(np.int32)
    return (magnitude[np.abs(values)] | np.where(values < 0, 0x80, 0)).astype(np.uint8)


def test_widen_codes_matches_e4m3_table(qi):
    rng = np.random.default_rng(91)
    rows, k = 96, 640
    codes = rng.integers(0, 256, size=(rows, k // 2), dtype=np.uint8)  # includes -8
    out = torch.zeros(rows, k, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_widen_codes_ex(up(codes), out, rows, k) == 0
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), e4m3_of_codes(codes))


@pytest.mark.parametrize("rows,k", [(1, 32), (33, 992), (16, 1024), (3, 5472)])  # around 16384 codes a block
def test_widen_codes_at_the_edges_of_its_blocks(qi, rows, k):
    codes = np.random.default_rng(92 + rows).integers(0, 256, size=(rows, k // 2), dtype=np.uint8)
    out = torch.full((rows * k + 64,), 0xAB, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_widen_codes_ex(up(codes), out, rows, k) == 0
    torch.cuda.synchronize()
    assert np.array_equal(out[:rows * k].cpu().numpy().reshape(rows, k), e4m3_of_codes(codes))
    assert bool((out[rows * k:] == 0xAB).all())


@pytest.mark.parametrize("m,n,k", [(1, 32, 512), (1, 32, 768), (5, 96, 1024), (300, 32, 768), (17, 288, 4096)])
def test_w4a4_packed_few_rows_or_outputs_by_shape(qi, m, n, k):
    rng = np.random.default_rng(94 + m + n + k)
    w_codes, w_scales = qt.pack_w4a4(qt.make_weights(rng, n, k))
    a_codes, a_scales = qo.quantize_activations(qt.make_activations(rng, m, k))
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm_ex(up(a_codes), up(a_scales), up(w_codes), up(w_scales), None, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(y.cpu().numpy(), qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales))


def test_a_refused_launch_is_reported_once(qi):
    # the legacy stream takes no launch while another stream that waits for it is captured: the call says so, and the next
    # call's status is its own
    runtime, on, graph = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(), ctypes.c_void_p()
    x, out = torch.ones(1024, device="cuda"), torch.zeros(4096, dtype=torch.float16, device="cuda")
    codes, halves = torch.zeros(64 * 32, dtype=torch.uint8, device="cuda"), torch.zeros(64, dtype=torch.float16, device="cuda")
    assert qi.f32_to_f16(x, out, 1024) == 0
    check_status(qi)
    assert runtime.cudaStreamCreateWithFlags(ctypes.byref(on), 0) == 0 and runtime.cudaStreamBeginCapture(on, 0) == 0
    refused = qi.f32_to_f16(x, out, 1024)
    ended = runtime.cudaStreamEndCapture(on, ctypes.byref(graph))
    runtime.cudaGetLastError()
    following = qi.w4a16_dequantize_ex(codes, halves, halves, out, 64, 64)
    assert runtime.cudaStreamDestroy(on) == 0
    assert (refused, ended, following) == (906, 901, 0)  # implicit use of the legacy stream, capture invalidated, success
    check_status(qi)


@pytest.mark.parametrize("m,n,k", [(1, 32, 768), (77, 96, 1024)])
def test_w4a4_packed_few_rows_captured(qi, m, n, k):
    # a captured call of few rows is one kernel without scratch: its graph can be instantiated more than once
    rng = np.random.default_rng(96 + m + n + k)
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    args = (up(a_codes), up(a_scales), up(w_codes), up(w_scales), None)
    y = torch.full((m, n), float("nan"), device="cuda")
    assert qi.w4a4_gemm_ex(*args, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    stream, runtime = torch.cuda.Stream(), ctypes.CDLL("libcudart.so.12")
    on, graph, first, second = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    captured = torch.full((m, n), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert runtime.cudaStreamBeginCapture(on, 0) == 0
    status = qi.w4a4_gemm_ex(*args, captured, qi.DTYPE_F32, n, m, n, k, stream.cuda_stream)
    assert runtime.cudaStreamEndCapture(on, ctypes.byref(graph)) == 0 and status == 0
    instances = [runtime.cudaGraphInstantiate(ctypes.byref(instance), graph, ctypes.c_ulonglong(0)) for instance in (first, second)]
    runtime.cudaGetLastError()
    assert instances == [0, 0]
    for instance in (first, second):
        captured.fill_(float("nan"))
        torch.cuda.synchronize()
        assert runtime.cudaGraphLaunch(instance, on) == 0
        check_status(qi)
        assert torch.equal(captured, y)
        assert runtime.cudaGraphExecDestroy(instance) == 0
    assert runtime.cudaGraphDestroy(graph) == 0
    assert np.array_equal(y.cpu().numpy(), qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales))


@pytest.mark.parametrize("m,n,k", [(1, 32, 256), (16, 4000, 512), (17, 3072, 1024), (33, 9216, 256), (77, 9216, 512), (96, 9248, 256), (130, 3072, 512), (77, 12288, 256), (256, 3072, 768),
                                   (33, 4768, 768), (40, 5024, 512), (48, 6272, 1024)])  # the last three in tiles of 16 rows
def test_w4a4_wide_few_rows_as_columns(qi, m, n, k):
    rng = np.random.default_rng(95 + m + n + k)
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    bias = qt.make_bias(rng, n)
    expected = qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales, bias=bias)
    args = (up(e4m3_of_codes(a_codes)), up(a_scales), up(e4m3_of_codes(w_codes)), up(w_scales), up(bias))
    y = torch.full((m + 1, n), float("nan"), dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm_wide_ex(*args, y, qi.DTYPE_F32, n, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(y[:m].cpu().numpy(), expected) and bool(torch.isnan(y[m]).all())
    y16 = torch.zeros(m, n, dtype=torch.float16, device="cuda")
    assert qi.w4a4_gemm_wide_ex(*args, y16, qi.DTYPE_F16, n, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(y16.cpu().numpy(), expected.astype(np.float16))


@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_quantize_wide_writes_the_same_codes_as_bytes(qi, dtype):
    rng = np.random.default_rng(93)
    m, k = 300, 1024
    x16 = qt.make_activations(rng, m, k)
    x = x16 if dtype == "f16" else x16.astype(np.float32)
    codes = torch.zeros(m, k // 2, dtype=torch.uint8, device="cuda")
    scales = torch.zeros(m, k // 64, dtype=torch.float16, device="cuda")
    wide = torch.zeros(m, k, dtype=torch.uint8, device="cuda")
    x_dtype = qi.DTYPE_F16 if dtype == "f16" else qi.DTYPE_F32
    assert qi.w4a4_quantize_activations_wide_ex(up(x), x_dtype, codes, scales, wide, m, k) == 0
    torch.cuda.synchronize()
    expected_codes, expected_scales = qo.quantize_activations(x)
    assert np.array_equal(codes.cpu().numpy(), expected_codes)
    assert np.array_equal(half_bits(scales), expected_scales)
    assert np.array_equal(wide.cpu().numpy(), e4m3_of_codes(expected_codes))
    wide2 = torch.zeros(m, k, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_quantize_activations_wide_ex(up(x), x_dtype, None, scales, wide2, m, k) == 0  # bytes only
    torch.cuda.synchronize()
    assert torch.equal(wide, wide2)


class WideKernel:
    """The byte-operand entry points, by shape or held to 128 x 128 tiles, behind the same two calls."""

    def __init__(self, qi, single):
        self.qi, self.single = qi, single

    def gemm(self, a, sa, w, sw, bias, y, y_dtype, ldy, m, n, k):
        if self.single:
            return self.qi.w4a4_gemm_wide_single_ex(a, sa, w, sw, bias, y, y_dtype, ldy, None, m, n, k)
        return self.qi.w4a4_gemm_wide_ex(a, sa, w, sw, bias, y, y_dtype, ldy, m, n, k)

    def group_dots(self, a, sa, w, sw, y, dots, m, n, k):
        if self.single:
            return self.qi.w4a4_gemm_wide_single_ex(a, sa, w, sw, None, y, self.qi.DTYPE_F32, n, dots, m, n, k)
        return self.qi.w4a4_group_dots_wide_ex(a, sa, w, sw, y, dots, m, n, k)


@pytest.fixture(params=["by shape", "128x128"])
def wide_kernel(request, qi):
    """The tiles that the shape takes (with the groups' dots: 256 x 128 on CTA pairs), and 128 x 128 tiles."""
    return WideKernel(qi, request.param == "128x128")


@pytest.mark.parametrize("m,n,k", [(128, 128, 128), (256, 384, 512), (128, 256, 3072), (200, 160, 1280),
                                   (640, 768, 256)])
def test_w4a4_wide_gemm_bits_and_exact_dots(qi, wide_kernel, m, n, k):
    rng = np.random.default_rng(5000 + m + n + k)
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    a_wide, w_wide = (torch.zeros(r, k, dtype=torch.uint8, device="cuda") for r in (m, n))
    assert qi.w4a4_widen_codes_ex(up(a_codes), a_wide, m, k) == 0
    assert qi.w4a4_widen_codes_ex(up(w_codes), w_wide, n, k) == 0
    y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    dots = torch.full((m, n, k // 64), 12345, dtype=torch.int32, device="cuda")
    args = (a_wide, up(a_scales), w_wide, up(w_scales))
    assert wide_kernel.group_dots(*args, y, dots, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(dots.cpu().numpy(), qo.w4a4_group_dots(a_codes, w_codes))
    expected = qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales)
    assert np.array_equal(y.cpu().numpy(), expected)
    bias = qt.make_bias(rng, n)
    y16 = torch.zeros(m, n, dtype=torch.float16, device="cuda")
    assert wide_kernel.gemm(*args, up(bias), y16, qi.DTYPE_F16, n, m, n, k) == 0
    check_status(qi)
    distance, checked = qt.fp16_store_error(y16.cpu().numpy(), qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales, bias=bias))
    assert distance <= FP16_STORE_ULPS and checked > 0.25


@pytest.mark.parametrize("m,n,k", [(2304, 2048, 1024), (1000, 1280, 3072), (4096, 3072, 640), (333, 4224, 2048),
                                   (2048, 1152, 12288)])
def test_w4a4_wide_gemm_equals_packed_kernel_on_many_tiles(qi, wide_kernel, m, n, k):
    # Shapes with more tiles than CTAs, ragged row counts and long K: CTAs walk several tiles and the
    # pipelines wrap many times. The byte-operand kernels must give the bits of the int8 kernel, launch after launch.
    generator = torch.Generator(device="cuda").manual_seed(m + n + k)
    def signed_codes(rows):
        v = torch.randint(-7, 8, (rows, k), dtype=torch.int16, device="cuda", generator=generator) & 0xF
        return (v[:, 0::2] | (v[:, 1::2] << 4)).to(torch.uint8).contiguous()
    a_codes, w_codes = signed_codes(m), signed_codes(n)
    a_scales = (torch.rand(m, k // 64, device="cuda", generator=generator) * 0.5 + 0.05).half()
    w_scales = (torch.rand(n, k // 64, device="cuda", generator=generator) * 5e-3 + 1e-3).half()
    a_wide, w_wide = (torch.zeros(r, k, dtype=torch.uint8, device="cuda") for r in (m, n))
    assert qi.w4a4_widen_codes_ex(a_codes, a_wide, m, k) == 0
    assert qi.w4a4_widen_codes_ex(w_codes, w_wide, n, k) == 0
    expected = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm_path_ex(a_codes, a_scales, w_codes, w_scales, None, expected, qi.DTYPE_F32, n, m, n, k, qi.W4A4_PATH_INT8) == 0
    check_status(qi)
    for _ in range(4):
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        assert wide_kernel.gemm(a_wide, a_scales, w_wide, w_scales, None, y, qi.DTYPE_F32, n, m, n, k) == 0
        check_status(qi)
        assert torch.equal(y, expected)


@pytest.mark.parametrize("m,n,k", [(1024, 4096, 256), (4096, 3072, 256), (300, 3072, 512), (1500, 2112, 256), (256, 32, 256), (2048, 9600, 256),
                                   (1, 32, 256), (16, 96, 512), (17, 9216, 256), (77, 3104, 1280), (129, 2048, 768), (300, 480, 2304)])
def test_w4a4_wide_gemm_in_narrow_tiles(qi, m, n, k):
    # last waves cut into narrower tiles, and few rows or outputs, against the int8 kernel; float16 into a slice of a wider matrix
    # with a bias, and float32
    rng = np.random.default_rng(m + n + k)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.02, 0.2)
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 0.002, 0.01)
    a, sa, w, sw = up(a_codes), up(a_scales.view(np.float16)), up(w_codes), up(w_scales.view(np.float16))
    bias = up(qt.make_bias(rng, n))
    a_wide = torch.empty(m, k, dtype=torch.uint8, device="cuda")
    w_wide = torch.empty(n, k, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_widen_codes_ex(a, a_wide, m, k) == 0 and qi.w4a4_widen_codes_ex(w, w_wide, n, k) == 0
    for dtype, code in ((torch.float32, qi.DTYPE_F32), (torch.float16, qi.DTYPE_F16)):
        ldy = n + 8
        got, expected = (torch.full((m, ldy), -7.0, dtype=dtype, device="cuda") for _ in range(2))
        assert qi.w4a4_gemm_wide_ex(a_wide, sa, w_wide, sw, bias, got, code, ldy, m, n, k) == 0
        assert qi.w4a4_gemm_path_ex(a, sa, w, sw, bias, expected, code, ldy, m, n, k, qi.W4A4_PATH_INT8) == 0
        check_status(qi)
        assert torch.equal(got, expected)


def random_wide_operands(qi, m, n, k):
    """Packed and byte-wide codes and scales of both operands, made on the device."""
    generator = torch.Generator(device="cuda").manual_seed(m + n + k)
    operands = []
    for rows, low, high in ((m, 0.05, 0.5), (n, 1e-3, 6e-3)):
        values = torch.randint(-7, 8, (rows, k), dtype=torch.int16, device="cuda", generator=generator) & 0xF
        codes = (values[:, 0::2] | (values[:, 1::2] << 4)).to(torch.uint8).contiguous()
        scales = (torch.rand(rows, k // 64, device="cuda", generator=generator) * (high - low) + low).half()
        wide = torch.empty(rows, k, dtype=torch.uint8, device="cuda")
        assert qi.w4a4_widen_codes_ex(codes, wide, rows, k) == 0
        operands.append((codes, wide, scales))
    return operands


# Few rows or outputs, one row past what each kind of tiles covers in a wave of 148 CTAs, several waves, rows and columns that end within a tile.
NARROW_SHAPES = [("16 rows", 6, 32, 512), ("16 rows", 130, 672, 512), ("32 rows", 19, 9568, 256), ("32 rows", 63, 9568, 256), ("48 rows", 40, 9568, 256),
                 ("48 rows", 99, 9568, 512), ("48 rows", 600, 2336, 512), ("128x32", 1209, 160, 256), ("128x32", 519, 1888, 256), ("128x64", 97, 6368, 256), ("128x64", 293, 5728, 256)]
# 256 x 64 tiles: a wave alone, whole or of 16, 32 or 48 columns; last waves of 16, 32, 48 and 64 columns; blocks of rows of tiles (74 MB of
# activations and more), the last one as high as the others (9000 rows), lower (8900), or shorter than the last wave, which then stays whole (9300).
TALL_SHAPES = [(200, 7712, 256), (511, 9248, 256), (252, 9600, 256), (385, 6304, 256), (294, 8160, 256), (247, 6304, 256), (1000, 3104, 512), (2049, 6016, 256),
               (1024, 12288, 256), (1000, 1280, 3072), (9000, 640, 8192), (8900, 640, 8192), (9300, 640, 8192)]


def test_the_shapes_of_the_tile_tests_take_the_tiles_that_they_name(qi):
    for tiles, *shape in NARROW_SHAPES:
        assert qi.w4a4_gemm_plan(*shape).tiles == tiles, shape
    plans = [qi.w4a4_gemm_plan(*shape) for shape in TALL_SHAPES]
    assert {plan.tiles for plan in plans} == {"256x64"}
    assert {(plan.whole > 0, plan.width) for plan in plans if plan.cut} >= {(False, 48), (True, 16), (True, 32), (True, 48)}
    assert {plan.whole % 148 > 0 for plan in plans if not plan.cut} == {True}
    assert [(plan.block, plan.last_rows, plan.cut > 0) for plan in plans[-3:]] == [(12, 12, True), (12, 11, True), (12, 1, False)]


@pytest.mark.parametrize("m,n,k", [tuple(shape) for _, *shape in NARROW_SHAPES] + TALL_SHAPES)
def test_w4a4_wide_gemm_in_each_kind_of_tiles(qi, m, n, k):
    # the bits of the int8 kernel; rows that start on 32 bytes (whole sectors to store) and rows that start on 16
    (a, a_wide, sa), (w, w_wide, sw) = random_wide_operands(qi, m, n, k)
    bias = torch.randn(n, device="cuda")
    for dtype, code, half_sector in ((torch.float32, qi.DTYPE_F32, 4), (torch.float16, qi.DTYPE_F16, 8)):  # elements of 16 bytes
        for ldy, start in ((n, 0), (n + half_sector, 0), (n, half_sector)):
            got, expected = (torch.full((m * ldy + 2 * half_sector,), -7.0, dtype=dtype, device="cuda") for _ in range(2))
            assert qi.w4a4_gemm_wide_ex(a_wide, sa, w_wide, sw, bias, got[start:], code, ldy, m, n, k) == 0
            assert qi.w4a4_gemm_path_ex(a, sa, w, sw, bias, expected[start:], code, ldy, m, n, k, qi.W4A4_PATH_INT8) == 0
            check_status(qi)
            assert torch.equal(got, expected)


@pytest.mark.parametrize("k", [512, 768])
def test_w4a4_tall_tiles_scales_from_eight_bytes(qi, k):
    # scales are read sixteen bytes at a time where rows begin on sixteen (an even number of four groups) and the arrays do, else eight
    m, n = 1000, 3104
    assert qi.w4a4_gemm_plan(m, n, k).tiles == "256x64"
    (a, a_wide, sa), (w, w_wide, sw) = random_wide_operands(qi, m, n, k)
    later_sa, later_sw = (torch.cat([t.flatten()[:4], t.flatten()])[4:] for t in (sa, sw))
    assert later_sa.data_ptr() % 16 == later_sw.data_ptr() % 16 == 8
    expected = torch.full((m, n), -7.0, device="cuda")
    assert qi.w4a4_gemm_path_ex(a, sa, w, sw, None, expected, qi.DTYPE_F32, n, m, n, k, qi.W4A4_PATH_INT8) == 0
    for row_scales, column_scales in ((sa, sw), (later_sa, sw), (sa, later_sw)):
        got = torch.full((m, n), -7.0, device="cuda")
        assert qi.w4a4_gemm_wide_ex(a_wide, row_scales, w_wide, column_scales, None, got, qi.DTYPE_F32, n, m, n, k) == 0
        check_status(qi)
        assert torch.equal(got, expected)


def test_w4a4_wide_gemm_extreme_dots(qi, wide_kernel):
    # all codes +-7: every group dot is +-3136, the largest the format allows; fp32 accumulation must stay exact
    m, n, k = 128, 128, 512
    a_codes = np.full((m, k // 2), 0x77, dtype=np.uint8)
    a_codes[1::2] = 0x99
    w_codes = np.full((n, k // 2), 0x77, dtype=np.uint8)
    w_codes[2::3] = 0x99
    w_codes[5::7] = 0x97
    ones = np.full((m, k // 64), np.float16(1.0)).view(np.uint16)
    a_wide, w_wide = (torch.zeros(r, k, dtype=torch.uint8, device="cuda") for r in (m, n))
    assert qi.w4a4_widen_codes_ex(up(a_codes), a_wide, m, k) == 0
    assert qi.w4a4_widen_codes_ex(up(w_codes), w_wide, n, k) == 0
    y = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    dots = torch.zeros(m, n, k // 64, dtype=torch.int32, device="cuda")
    assert wide_kernel.group_dots(a_wide, up(ones), w_wide, up(ones[:n]), y, dots, m, n, k) == 0
    check_status(qi)
    expected = qo.w4a4_group_dots(a_codes, w_codes)
    assert np.abs(expected).max() == 3136
    assert np.array_equal(dots.cpu().numpy(), expected)


def test_linear_takes_the_wide_path_when_given_wide_operands(qi):
    rng = np.random.default_rng(95)
    rows, n, k = 256, 384, 768
    x32 = qt.make_activations(rng, rows, k).astype(np.float32)
    codes, scales = qt.pack_w4a4(qt.make_weights(rng, n, k))
    wide_w = torch.zeros(n, k, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_widen_codes_ex(up(codes), wide_w, n, k) == 0
    work = qi.LinearWork(torch.zeros(rows * k // 2, dtype=torch.uint8, device="cuda"),
                         torch.zeros(rows * k // 64, dtype=torch.float16, device="cuda"),
                         torch.zeros(rows * k, dtype=torch.float16, device="cuda"),
                         wide=torch.zeros(rows * k, dtype=torch.uint8, device="cuda"))
    record = qi.PackedLinear(qi.SCHEME_W4A4_H256, n, k, up(codes), up(scales), weights_wide=wide_w)
    y = torch.zeros(rows, n, dtype=torch.float32, device="cuda")
    assert qi.linear(record, work, up(x32), y, rows) == 0
    check_status(qi)
    a_codes, a_scales = qo.quantize_activations(x32)
    assert np.array_equal(y.cpu().numpy(), qo.w4a4_gemm(a_codes, a_scales, codes, scales))
    assert work.wide.abs().sum().item() > 0  # the byte arena was really used


# ---- a wait that runs out ------------------------------------------------------------------------------

def test_a_wait_that_runs_out_reports_its_code_and_leaves_the_device_healthy(qi):
    # every device-side wait of the library is bounded; this makes one run out on purpose (a barrier nothing
    # arrives on, limit 1 ms, in a warp of which every other lane waits for nothing: the lanes have to give up
    # together, another code says they did not) and follows the error path a caller would see: code set, cleared
    # by reading it, and the next launches unaffected
    assert qi.kernel_status() == 0
    assert qi.probe_wait_timeout(1_000_000) == 0
    torch.cuda.synchronize()
    code = qi.kernel_status()
    assert code == 0x0001A000, hex(code)
    assert qi.kernel_status() == 0  # reading clears it
    assert qi.probe_wait_timeout(0) == qi.CUDA_ERROR_INVALID_VALUE
    assert qi.probe_wait_timeout(10**9) == qi.CUDA_ERROR_INVALID_VALUE
    rng = np.random.default_rng(808)
    m, n, k = 256, 256, 512
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    y = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    assert qi.w4a4_gemm(up(a_codes), up(a_scales), up(w_codes), up(w_scales), y, m, n, k) == 0
    check_status(qi)
    assert np.array_equal(y.cpu().numpy(), qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales))


# 256 x 128 tiles on 74 pairs of CTAs: two and three tiles a pair, rows and columns that end within a tile, one stage of K and rings that wrap.
@pytest.mark.parametrize("m,n,k", [(2304, 2048, 1024), (5000, 1056, 768), (700, 4128, 2304), (2048, 1152, 12288), (2300, 2080, 256)])
def test_w4a4_scatter_over_several_tiles(qi, m, n, k):
    # into two local buffers as the copies, beside what else stands in their rows: the bits of the int8 kernel
    (a, a_wide, sa), (w, w_wide, sw) = random_wide_operands(qi, m, n, k)
    ldy, column = n + 96, 64
    for bias in (None, torch.randn(n, device="cuda")):
        for dtype, code in ((torch.float32, qi.DTYPE_F32), (torch.float16, qi.DTYPE_F16)):
            expected = torch.full((m, ldy), -3.0, dtype=dtype, device="cuda")
            assert qi.w4a4_gemm_path_ex(a, sa, w, sw, bias, expected[:, column:], code, ldy, m, n, k, qi.W4A4_PATH_INT8) == 0
            outputs = [torch.full((m, ldy), -3.0, dtype=dtype, device="cuda") for _ in range(2)]
            copies = (ctypes.c_void_p * 2)(*[t.data_ptr() for t in outputs])
            assert qi.w4a4_gemm_wide_scatter_ex(a_wide, sa, w_wide, sw, bias, copies, 1, code, ldy, column, m, n, k) == 0
            check_status(qi)
            assert all(torch.equal(output, expected) for output in outputs)


def test_w4a4_group_dots_over_several_tiles(qi):
    m, n, k = 2100, 2080, 512  # 153 tiles on 74 pairs
    (a, a_wide, sa), (w, w_wide, sw) = random_wide_operands(qi, m, n, k)
    y, expected = (torch.full((m, n), float("nan"), device="cuda") for _ in range(2))
    dots, expected_dots = (torch.full((m, n, k // 64), 12345, dtype=torch.int32, device="cuda") for _ in range(2))
    assert qi.w4a4_group_dots_wide_ex(a_wide, sa, w_wide, sw, y, dots, m, n, k) == 0
    assert qi.w4a4_group_dots_ex(a, sa, w, sw, expected, expected_dots, m, n, k) == 0
    check_status(qi)
    assert torch.equal(dots, expected_dots) and torch.equal(y, expected)


@pytest.mark.parametrize("dtype_name", ["f16", "f32"])
def test_w4a4_scatter_epilogue_keeps_inside_a_slice_that_ends_within_a_tile(qi, dtype_name):
    """The GEMM that stores its slice into several copies of the whole output, on one GPU with two local buffers as the
    copies: n = 160 ends inside the kernel's 128-column tile, so the tile's last 96 columns must not be written. Canary
    values around the slice, in every copy, stay as they were."""
    import ctypes
    rng = np.random.default_rng(8100)
    m, n, k, ldy, column = 256, 160, 512, 512, 32
    w_codes, w_scales = qt.random_w4a4_pack(rng, n, k, 1e-3, 6e-3)
    a_codes, a_scales = qt.random_w4a4_pack(rng, m, k, 0.05, 0.6)
    expected = qo.w4a4_gemm(a_codes, a_scales, w_codes, w_scales)
    a_wide = torch.zeros(m, k, dtype=torch.uint8, device="cuda")
    w_wide = torch.zeros(n, k, dtype=torch.uint8, device="cuda")
    assert qi.w4a4_widen_codes_ex(up(a_codes), a_wide, m, k) == 0
    assert qi.w4a4_widen_codes_ex(up(w_codes), w_wide, n, k) == 0
    dtype, torch_dtype = (qi.DTYPE_F16, torch.float16) if dtype_name == "f16" else (qi.DTYPE_F32, torch.float32)
    outputs = [torch.full((m, ldy), -3.0, dtype=torch_dtype, device="cuda") for _ in range(2)]
    copies = (ctypes.c_void_p * 2)(*[t.data_ptr() for t in outputs])
    assert qi.w4a4_gemm_wide_scatter_ex(a_wide, up(a_scales), w_wide, up(w_scales), None, copies, 1, dtype, ldy, column,
                                        m, n, k) == 0
    torch.cuda.synchronize()
    check_status(qi)
    for output in outputs:
        got = output.float().cpu().numpy()
        assert np.all(got[:, :column] == -3.0) and np.all(got[:, column + n:] == -3.0)
        if dtype == qi.DTYPE_F32:
            assert np.array_equal(got[:, column:column + n], expected)
        else:
            distance, checked = qt.fp16_store_error(output[:, column:column + n].cpu().numpy(), expected)
            assert distance <= FP16_STORE_ULPS and checked > 0.5

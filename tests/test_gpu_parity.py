"""Parity of the CUDA kernels with the CPU oracle, through the C ABI, on a B200.

Bars (from the operator's definition): activation codes and scales, unpacked weights and
per-group integer dots bit-exact; fp32 outputs within 1e-3 of max|y|; fp16 stores within
2 fp16 ulp of the fp32 oracle rounded to fp16."""
import ctypes

import numpy as np
import pytest

import __graft_entry__ as entry
from oracle import qipack_oracle as qo
from tests import qi_testing as qt

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OUTPUT_TOLERANCE = 1e-3  # max |y - oracle| / max |oracle|, fp32 accumulate
FP16_STORE_ULPS = 2


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

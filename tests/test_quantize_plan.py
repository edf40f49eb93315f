"""Which form the plain activation quantiser takes: host code, no GPU."""
import os

import pytest

import __graft_entry__ as entry


@pytest.fixture(scope="module")
def qi():
    module = entry.load_package()
    if not os.path.exists(module.LIB_PATH):
        module.build()
    return module


@pytest.mark.parametrize("sms", [148, 74, 132])
def test_the_limits_are_chunks_per_multiprocessor(qi, sms):
    # a limit for each form, the last chunk count below it and the first above, on GPUs of different sizes
    for limit, below, above in ((8, 32, 64), (21, 64, 0), (48, 0, 256), (222, 256, 0)):
        assert qi.w4a4_quantize_plan(limit * sms, 256, sms).threads == below
        assert qi.w4a4_quantize_plan(limit * sms + 1, 256, sms).threads == above


# Microseconds on B200 of the linear with the paired form and with eight warps a CTA, another matrix of weights every launch.
@pytest.mark.parametrize("shape,paired,eight", [
    ((600, 1024, 3072), 14.2, 15.0), ((501, 1248, 4608), 18.09, 18.95), ((900, 1024, 2048), 14.4, 15.0), ((176, 832, 10496), 21.7, 22.4), ((488, 704, 4096), 17.6, 18.5),
    ((600, 3072, 3072), 21.1, 19.8), ((500, 3072, 4096), 23.9, 22.9), ((900, 12288, 2048), 56.5, 55.6), ((600, 1024, 4096), 19.2, 19.4), ((800, 3072, 3072), 31.3, 30.2),
], ids=str)
def test_the_faster_form_stands_in_front_of_a_linears_gemm(qi, shape, paired, eight):
    m, n, k = shape
    chosen = {0: paired, 256: eight}[qi.w4a4_quantize_plan(m, k, n=n).threads]
    assert chosen <= min(paired, eight) * 1.015  # a drawn shape varies by a percent


def test_one_round_of_the_paired_form_is_for_narrow_tiles_alone(qi):
    for m, narrow in ((445, 0), (592, 0), (593, 256)):  # 7120, 9472 and 9488 chunks; 48 and 64 on each of 148 multiprocessors are 7104 and 9472
        assert qi.w4a4_gemm_plan(m, 896, 4096).tiles != "256x64" and qi.w4a4_gemm_plan(m, 3072, 4096).tiles == "256x64"
        assert [qi.w4a4_quantize_plan(m, 4096, n=n).threads for n in (896, 3072, 0)] == [narrow, 256, 256]


# Microseconds likewise with the paired form and with two and four warps a CTA.
@pytest.mark.parametrize("shape,paired,two,four", [
    ((94, 1504, 6144), 13.69, 15.16, 12.73), ((50, 3072, 12288), 25.3, 26.7, 25.4), ((116, 1024, 6144), 13.3, 14.8, 12.5), ((100, 6144, 6144), 20.9, 21.6, 20.1),
    ((75, 6144, 8192), 24.2, 25.5, 23.5), ((68, 5216, 11264), 24.5, 26.7, 23.9), ((132, 1024, 5120), 12.05, 12.44, 11.05), ((86, 1120, 8704), 15.2, 16.6, 14.6),
    ((300, 3072, 2048), 13.75, 12.6, 13.03), ((256, 1024, 3072), 10.89, 9.96, 10.36), ((200, 3072, 3072), 13.75, 12.93, 13.12), ((170, 3072, 3072), 12.3, 11.4, 11.9),
], ids=str)
def test_long_rows_take_more_warps(qi, shape, paired, two, four):
    m, n, k = shape
    chosen = {0: paired, 64: two, 128: four}[qi.w4a4_quantize_plan(m, k, n=n).threads]
    assert chosen <= min(paired, two, four) * 1.015


def test_the_limits_of_four_warps(qi):
    # 14 and 21 chunks on each of 148 multiprocessors, in rows of 16 and of 17 chunks and of 256 inputs
    for m, k, threads in ((129, 4096, 64), (194, 4096, 64), (195, 4096, 0), (121, 4352, 64), (122, 4352, 128), (182, 4352, 128), (183, 4352, 0)):
        assert qi.w4a4_quantize_plan(m, k).threads == threads, (m, k)


@pytest.mark.parametrize("m,k", [(0, 256), (1, 0), (1, 128), (-1, 256)])
def test_no_plan_for_what_the_quantiser_refuses(qi, m, k):
    with pytest.raises(ValueError):
        qi.w4a4_quantize_plan(m, k)

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


@pytest.mark.parametrize("m,k", [(0, 256), (1, 0), (1, 128), (-1, 256)])
def test_no_plan_for_what_the_quantiser_refuses(qi, m, k):
    with pytest.raises(ValueError):
        qi.w4a4_quantize_plan(m, k)

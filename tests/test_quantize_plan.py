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


@pytest.mark.parametrize("m,k", [(0, 256), (1, 0), (1, 128), (-1, 256)])
def test_no_plan_for_what_the_quantiser_refuses(qi, m, k):
    with pytest.raises(ValueError):
        qi.w4a4_quantize_plan(m, k)

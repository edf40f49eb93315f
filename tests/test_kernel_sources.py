"""Rules of the kernel sources that a run cannot show: a hand-over that is one barrier short gives wrong sums only now and then."""
import glob
import os
import re

import pytest

import __graft_entry__ as entry

KERNELS = sorted(glob.glob(os.path.join(entry.PACKAGE_DIR, "csrc", "*.cuh")))


def statements(path):
    """The file's lines without comments and blank ones, as (number, text)."""
    lines = (re.sub(r"//.*", "", line).strip() for line in open(path, encoding="utf-8"))
    return [(number, line) for number, line in enumerate(lines, 1) if line]


@pytest.mark.parametrize("path", KERNELS, ids=os.path.basename)
def test_a_lane_that_arrives_for_its_warp_follows_a_warp_barrier(path):
    # lane 0's arrival says that ALL lanes have read or written what changes hands; only a __syncwarp() orders theirs before it
    code = statements(path)
    for i, (number, line) in enumerate(code):
        if not line.startswith("if (lane == 0)"):
            continue
        first = code[i + 1][1] if line.endswith("{") else line
        if "arrive" in first and "expect_tx" not in first:
            assert code[i - 1][1] == "__syncwarp();", f"{os.path.basename(path)}:{number}: arrives for lanes that may not be there yet"


def test_the_rule_reaches_the_hand_overs():
    arrivals = sum(line.startswith("if (lane == 0)") and "arrive" in line for path in KERNELS for _, line in statements(path))
    assert arrivals >= 15


def test_tmem_is_taken_before_the_next_kernel_may_start():
    # else a CTA could wait for TMEM that a later kernel's CTA holds, which waits for this one's kernel to end; and no two CTAs
    # that wait for others of their clusters may share an SM (both conditions: beside grid_release)
    kernels = clusters = 0
    for path in KERNELS:
        source = "\n".join(line for _, line in statements(path))
        for kernel in re.split(r"__global__", source)[1:]:
            taken = kernel.find("tmem_alloc")
            if taken < 0 or "grid_wait()" not in kernel:
                continue
            kernels += 1
            assert "grid_release()" not in kernel[:taken], os.path.basename(path)
            if "cluster_sync()" in kernel:
                clusters += 1
                assert "ONE_CTA_SMEM" in source, os.path.basename(path)
    assert kernels >= 9 and clusters == 4


def test_every_source_makes_the_library_stale():
    # a kernel file that is not on the list could be edited without the library being built again
    assert sorted(entry.load_package().SOURCES) == sorted(os.listdir(os.path.join(entry.PACKAGE_DIR, "csrc")))

"""Which tiles the byte-operand W4A4 GEMM takes for a shape, and that its tiles cover the output: host code, no GPU."""
import os

import pytest

import __graft_entry__ as entry


@pytest.fixture(scope="module")
def qi():
    module = entry.load_package()
    if not os.path.exists(module.LIB_PATH):
        module.build()
    return module


# Microseconds on B200 of the kernels that come into question (148 SMs, another matrix of weights every launch).
MEASURED = {
    (264, 9568, 3328): {"256x64": 37.9, "128x64": 35.4, "32 rows": 32.6, "48 rows": 29.5},
    (308, 12288, 3072): {"256x64": 41.2, "128x64": 35.8, "128x32": 42.5, "48 rows": 35.1},
    (771, 3072, 3072): {"256x64": 24.5, "128x64": 28.2, "32 rows": 26.3, "48 rows": 22.0},
    (783, 5440, 1792): {"256x64": 25.0, "128x64": 28.9, "32 rows": 28.6, "48 rows": 23.4},
    (169, 9792, 768): {"256x64": 10.6, "128x64": 12.7, "32 rows": 10.7, "48 rows": 9.7},
    (593, 4096, 4096): {"256x64": 31.4, "128x64": 41.0, "32 rows": 43.0, "48 rows": 34.6},
    (708, 1568, 4096): {"256x64": 15.6, "128x64": 23.4, "128x32": 19.8, "48 rows": 23.8},
    (144, 6816, 12288): {"256x64": 45.1, "128x64": 73.7, "32 rows": 53.8, "48 rows": 64.5},
    (190, 8896, 9728): {"256x64": 42.0, "48 rows": 47.6},
    (401, 3072, 12288): {"256x64": 43.4, "128x64": 60.4, "48 rows": 60.0},
    (178, 5248, 8960): {"256x64": 31.6, "32 rows": 30.2, "48 rows": 33.8},
    (228, 576, 2560): {"256x64": 8.2, "128x64": 9.7, "128x32": 6.8, "16 rows": 5.4, "32 rows": 6.7},
    (13, 4096, 4096): {"128x32": 9.6, "16 rows": 9.7, "32 rows": 8.8, "48 rows": 9.7},
    (45, 3072, 12288): {"128x64": 28.9, "128x32": 21.5, "16 rows": 23.0, "32 rows": 27.4},
}


@pytest.mark.parametrize("shape", MEASURED, ids=lambda shape: "x".join(map(str, shape)))
def test_the_tiles_that_measure_fastest_are_taken(qi, shape):
    times = MEASURED[shape]
    chosen = qi.w4a4_gemm_plan(*shape).tiles
    # 5 %: the prices are within 2 to 6 % of the times, and one GPU's times within 2 % of another's
    assert chosen in times and times[chosen] <= 1.05 * min(times.values()), (chosen, times)

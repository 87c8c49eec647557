"""Block shapes of the 2-D morphology kernels (iane_gb300/csrc/plane_lanes.h): on narrow images too,
most of a block's threads have elements."""
from __future__ import annotations

import pytest

from host_code import compile_host

SOURCE = """
#include "plane_lanes.h"
extern "C" int lanes(int nx, int ny, int px, int rows, int aligned, int r)
{
	return iane_gb::plane_lanes(nx, ny, px, rows, aligned != 0, r);
}
"""


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    return compile_host(tmp_path_factory.mktemp("lanes"), SOURCE).lanes


@pytest.mark.parametrize("px,rows", [(4, 4), (8, 8)], ids=["f32", "integers"])
@pytest.mark.parametrize("aligned", [0, 1])
@pytest.mark.parametrize("r", [1, 4])
def test_threads_have_elements(lanes, px, rows, aligned, r):
    for nx in [*range(1, 140), 255, 256, 257, 300, 511, 513, 640, 1000, 1024, 1920, 2560]:
        for ny in (1, 40, 1080, 20000):
            n = lanes(nx, ny, px, rows, aligned, r)
            assert n in (1, 2, 4, 8, 16, 32)
            threads = -(-nx // (n * px)) * n          # side by side
            used = -(-nx // px)
            assert used > 0.5 * threads, (nx, ny, n)  # 2 of 32 used for 16 elements, 32 always side by side

"""Completion counters of the persistent Richardson-Lucy kernels (iane_gb300/csrc/counters.h) near
and beyond 2^31 and 2^32: an image's counter takes four completions per tile and phase, and a run of
2^31 items is accepted."""
from __future__ import annotations

import ctypes

import pytest

from host_code import compile_host

SOURCE = """
#include "counters.h"
extern "C" int reached(unsigned have, unsigned need) { return iane_gb::counter_reached(have, need); }
extern "C" unsigned need(int phase, int tiles) { return iane_gb::batch_need(phase, tiles); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    lib = compile_host(tmp_path_factory.mktemp("counters"), SOURCE)
    lib.need.argtypes, lib.need.restype = [ctypes.c_int, ctypes.c_int], ctypes.c_uint
    lib.reached.argtypes, lib.reached.restype = [ctypes.c_uint, ctypes.c_uint], ctypes.c_int
    return lib


# tiles of an image and its phases: 2^30 tile-phases are 2^32 completions, and items of four tiles
# pass the run's bound of 2^31 items with 2^33 tile-phases
@pytest.mark.parametrize("tiles,phases", [(1, 2), (1, 8192), (512 * 512, 4095), (512 * 512, 4096), (512 * 512, 8190),
                                          (375 * 375, 8192), (1 << 20, 8192), (262143, 2 * 4095)])
def test_a_tile_waits_for_exactly_its_image_s_previous_phase(rule, tiles, phases):
    for phase in sorted({p for p in (1, 2, phases // 2, phases // 2 + 1, (1 << 29) // tiles, (1 << 30) // tiles,
                                     (1 << 30) // tiles + 1, (1 << 31) // tiles, phases - 1) if 0 < p < phases}):
        want = 4 * tiles * phase  # completions, not reduced
        need = rule.need(phase, tiles)
        for have in (want, want + 1, want + 4 * tiles - 1):  # the phase in work, up to its last completion
            assert rule.reached(have & 0xFFFFFFFF, need), (phase, have)
        for have in (want - 1, want - 4 * min(tiles, 2432), max(0, want - 4 * tiles)):  # tiles of the phase before missing
            assert not rule.reached(have & 0xFFFFFFFF, need), (phase, have)

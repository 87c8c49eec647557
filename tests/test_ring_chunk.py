"""The split along z of the marching kernels (iane_gb300/csrc/ring_chunk.h): the best of every count of
chunks, without looking at each of thousands on tall volumes, where that took longer than the kernel."""
from __future__ import annotations

import ctypes
import math

import pytest

from host_code import compile_host

SOURCE = """
#include "ring_chunk.h"
extern "C" int chunk(long long columns, int nz, int r, long long slots, int* looked)
{
	return iane_gb::ring_chunk(columns, nz, r, slots, looked);
}
extern "C" int narrow(int nx, int most) { return iane_gb::ring_narrow(nx, most); }
"""


@pytest.fixture(scope="module")
def chunk(tmp_path_factory):
    lib = compile_host(tmp_path_factory.mktemp("chunk"), SOURCE)
    lib.chunk.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_void_p]
    return lib.chunk


def score(columns, nz, r, slots, zc):
    blocks = columns * -(-nz // zc)
    return blocks / slots / -(-blocks // slots) * zc / (zc + 2 * r)


@pytest.mark.parametrize("columns", [1, 3, 40, 128, 2000])
@pytest.mark.parametrize("nz", [1, 2, 7, 64, 100, 511, 4096, 20000])
@pytest.mark.parametrize("r,slots", [(1, 608), (2, 456), (4, 304)])
def test_the_best_length_of_all(chunk, columns, nz, r, slots):
    looked = ctypes.c_int(0)
    got = chunk(columns, nz, r, slots, ctypes.byref(looked))
    best, want = -1.0, nz
    for chunks in range(1, nz + 1):
        zc = -(-nz // chunks)
        s = score(columns, nz, r, slots, zc)
        if s > best + 1e-9:
            best, want = s, zc
        if columns * -(-nz // zc) / slots > 8:
            break
    assert got == want
    assert looked.value <= 2 * math.sqrt(nz) + 2


def test_no_half_of_a_warp_without_columns(tmp_path_factory):
    narrow = compile_host(tmp_path_factory.mktemp("narrow"), SOURCE).narrow
    for nx in range(16, 1200):
        columns = 64 if narrow(nx, 1 << 30) else 128
        assert -(-nx // columns) * columns - nx < 64, nx
        assert narrow(nx, 3) == (narrow(nx, 1 << 30) and nx <= 192)

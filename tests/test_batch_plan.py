"""The host side of the batched Richardson-Lucy run (iane_gb300/csrc/batch_plan.h)."""
from __future__ import annotations

import ctypes

import pytest

from host_code import compile_host

SOURCE = r"""
#include "batch_plan.h"

#include <cstring>

using namespace iane_gb;

static std::vector<int> list(const int* p, int n) { return std::vector<int>(p, p + n); }

extern "C" void key(const int* nx, const int* ny, const int* kx, const int* ky, int n, int sms, char* out)
{
	std::strcpy(out, tune_key(list(nx, n), list(ny, n), list(kx, n), list(ky, n), sms).c_str());
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    return compile_host(tmp_path_factory.mktemp("plan"), SOURCE)


def ints(values):
    return (ctypes.c_int * len(values))(*values)


def key_of(plan, nx, ny, kx, ky, sms):
    out = ctypes.create_string_buffer(200)
    plan.key(ints(nx), ints(ny), ints(kx), ints(ky), len(nx), sms, out)
    return out.value.decode()


def test_the_tuned_choice_s_key_names_its_version(plan):
    h = 1469598103934665603
    for v in (300, 40, 5, 7, 210, 200, 15, 15):
        for byte in v.to_bytes(4, "little"):
            h = (h ^ byte) * 1099511628211 % 2 ** 64
    got = key_of(plan, [300, 210], [40, 200], [5, 15], [7, 15], 152)
    before = f"rl2d-batch f32 images 2 shapes {h:x} sms 152"  # as long as orders and kernel were others
    assert got != before
    assert got == before.replace("rl2d-batch", "rl2d-batch v2")
    assert got != key_of(plan, [300, 210], [40, 200], [5, 15], [15, 15], 152)

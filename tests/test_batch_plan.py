"""The host side of the batched Richardson-Lucy run (iane_gb300/csrc/batch_plan.h): the tuned choice's
key, the work items, the queues and their SMs -- and, with these and the kernel's rule for its counters
(counters.h), a simulation of how its CTAs take, hand on and count tiles (rl_batch_kernel.cu)."""
from __future__ import annotations

import ctypes
import heapq
import random

import pytest

from host_code import compile_host

SOURCE = r"""
#include "batch_plan.h"
#include "counters.h"

#include <cstring>

using namespace iane_gb;

static std::vector<int> list(const int* p, int n) { return std::vector<int>(p, p + n); }

extern "C" void key(const int* nx, const int* ny, const int* kx, const int* ky, int n, int sms, char* out)
{
	std::strcpy(out, tune_key(list(nx, n), list(ny, n), list(kx, n), list(ky, n), sms).c_str());
}

// items as seven ints each; per queue first, count and SMs; the start table. Returns the number of items.
extern "C" int queues(const int* nx, const int* ny, const int* kx, const int* ky, int n, int order, int group, int sms,
	int* items, int* classes, int* first, int* count, float* cost, int* start)
{
	const auto list_nx = list(nx, n), list_ny = list(ny, n);
	const auto made = make_items(list_nx, list_ny, list(kx, n), list(ky, n), order, group);
	const BatchQueues q = make_queues(made, list_nx, list_ny, order, sms, sms);
	for (const BatchItem& i : made) {
		const int v[] = {i.image, i.x0, i.y0, i.count, i.image_tiles, i.kx, i.ky};
		std::memcpy(items, v, sizeof v);
		items += 7;
	}
	*classes = q.classes;
	for (int c = 0; c < q.classes; ++c) {
		first[c] = q.of[c].first;
		count[c] = q.of[c].count;
		cost[c] = q.of[c].cost;
	}
	for (int s = 0; s < q.sms; ++s) start[s] = q.start[s];
	return static_cast<int>(made.size());
}
extern "C" int reached(unsigned have, unsigned need) { return counter_reached(have, need); }
extern "C" unsigned need(int phase, int tiles) { return batch_need(phase, tiles); }
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


def queues_of(plan, images, order, group, sms):
    nx, ny, kx, ky = (ints(v) for v in zip(*images))
    tiles = sum(-(-a // 64) * -(-b // 64) for a, b, _, _ in images)
    items, classes = (ctypes.c_int * (7 * tiles))(), ctypes.c_int(0)
    first, count, cost, start = (ctypes.c_int * 16)(), (ctypes.c_int * 16)(), (ctypes.c_float * 16)(), (ctypes.c_int * sms)()
    n = plan.queues(nx, ny, kx, ky, len(images), order, group, sms, items, ctypes.byref(classes), first, count, cost, start)
    return ([tuple(items[7 * i:7 * i + 7]) for i in range(n)],
            [(first[c], count[c], cost[c]) for c in range(classes.value)], list(start))


def some_images(rng, n):
    return [(rng.randint(1, 400), rng.randint(1, 300), 2 * rng.randint(0, 15) + 1, 2 * rng.randint(0, 31) + 1) for _ in range(n)]


@pytest.mark.parametrize("group", [0, 1, 2, 3])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("n,sms", [(1, 152), (5, 3), (40, 152), (60, 7), (60, 148)])
def test_items_cover_the_batch_and_queues_share_the_sms(plan, n, sms, order, group):
    images = some_images(random.Random(n * 10 + order), n)
    items, queues, start = queues_of(plan, images, order, group, sms)
    seen = set()
    for image, x0, y0, count, tiles, kx, ky in items:
        nx, ny, wx, wy = images[image]
        assert (kx, ky, tiles) == (wx, wy, -(-nx // 64) * -(-ny // 64)) and count in (1, 2, 3, 4)
        for t in range(count):
            assert x0 + 64 * t < nx and y0 < ny and x0 % 64 == y0 % 64 == 0
            assert (image, x0 + 64 * t, y0) not in seen
            seen.add((image, x0 + 64 * t, y0))
    assert len(seen) == sum(-(-a // 64) * -(-b // 64) for a, b, _, _ in images)
    at = 0  # the queues are the list, in order, each of one width (or one of all)
    for first, count, cost in queues:
        assert first == at and count > 0 and cost > 0
        at += count
        if order == 1:
            assert len({i[5] for i in items[first:at]}) == 1
    assert at == len(items) and len(queues) == (len({i[5] for i in items}) if order == 1 else 1)
    assert all(0 <= c < len(queues) for c in start) and start == sorted(start)
    if sms >= len(queues):
        assert set(start) == set(range(len(queues)))  # an SM for every queue
        work = [count * cost for _, count, cost in queues]
        for c in range(len(queues)):  # and shares within one SM, but for queues raised to their first one
            assert start.count(c) <= max(1.0, work[c] / sum(work) * sms + 1)


def simulate(plan, images, order, group, sms, ctas_per_sm, phases, ahead, rng):
    """One run: every CTA has a tile in work and, with `ahead` or within an item, the next one in hand, as in
    batch_persistent_kernel."""
    items, queues, start = queues_of(plan, images, order, group, sms)
    heads, done, true_done = [0] * len(queues), [0] * len(images), {}
    finished = set()

    def take(cta):
        if cta["phase"] >= 0 and cta["next"] + 1 < cta["item"][3]:
            cta["next"] += 1
            return
        cls, cta["phase"] = cta["cls"], -1
        while cls >= 0:
            first, count, _ = queues[cls]
            k = heads[cls]
            heads[cls] += 1
            if k < count * phases:
                cta["phase"], cta["item"], cta["next"] = k // count, items[first + k % count], 0
                break
            left = [(count * phases - heads[c]) * cost if heads[c] < count * phases else -1.0
                    for c, (_, count, cost) in enumerate(queues)]
            cls = max(range(len(left)), key=left.__getitem__) if max(left) > 0 else -1
        cta["cls"] = cls

    def free(cta):
        item = cta["item"]
        return cta["phase"] <= 0 or plan.reached(done[item[0]], plan.need(cta["phase"], item[4]))

    def issue(cta):
        if cta["phase"] < 0:
            return None
        image, x0, y0, _, tiles, _, _ = cta["item"]
        p = cta["phase"]
        # its loads begin: the image's previous phase is complete, and nothing of the phase after this one is
        assert p == 0 or true_done.get((image, p - 1), 0) == 4 * tiles
        assert true_done.get((image, p + 1), 0) == 0
        return p, image, x0 + 64 * cta["next"], y0, tiles

    def run(cta):  # yields a delay, or None to be asked again
        take(cta)
        while not free(cta):
            yield None
        tile = issue(cta)
        while tile is not None:
            yield rng.uniform(0.0, 1.0)
            held = ahead or cta["next"] + 1 < cta["item"][3]
            if held:
                take(cta)
            yield rng.uniform(0.5, 3.0)  # landing and sums
            later, issued = not held or not free(cta), False
            if not later:
                tile_after, issued = issue(cta), True
            for _ in range(4):  # the warps' epilogues, each counting for itself
                yield rng.uniform(0.0, 0.5)
                done[tile[1]] += 1
                true_done[tile[1], tile[0]] = true_done.get((tile[1], tile[0]), 0) + 1
            assert tile[:4] not in finished
            finished.add(tile[:4])
            if not issued:
                if not held:
                    take(cta)
                while not free(cta):
                    yield None
                tile_after = issue(cta)
            tile = tile_after

    ctas = [{"phase": -1, "next": 0, "item": None, "cls": start[k % sms]} for k in range(ctas_per_sm * sms)]
    active, waiting = [], []
    now = 0.0
    for k, cta in enumerate(ctas):
        heapq.heappush(active, (rng.uniform(0.0, 1.0), k, run(cta)))
    while active:
        now, k, gen = heapq.heappop(active)
        for delay, (j, g) in [(0.0, (k, gen))] + [(0.0, w) for w in waiting]:
            try:
                step = next(g)
            except StopIteration:
                if (j, g) in waiting:
                    waiting.remove((j, g))
                continue
            if step is None:
                if (j, g) not in waiting:
                    waiting.append((j, g))
            else:
                if (j, g) in waiting:
                    waiting.remove((j, g))
                heapq.heappush(active, (now + step, j, g))
    assert not waiting, "stalled"
    tiles = sum(-(-a // 64) * -(-b // 64) for a, b, _, _ in images)
    assert len(finished) == phases * tiles


@pytest.mark.parametrize("group", [0, 2, 3])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("ahead", [False, True])
@pytest.mark.parametrize("sms,ctas_per_sm", [(1, 1), (2, 1), (3, 4), (40, 2)])
def test_tiles_in_work_and_in_hand_keep_the_order_and_end(plan, sms, ctas_per_sm, ahead, order, group):
    for seed in range(4):
        rng = random.Random(seed * 100 + sms)
        images = [(64 * rng.randint(1, 9), 64 * rng.randint(1, 3), rng.choice([1, 5, 5, 7, 15, 31]), 5)
                  for _ in range(rng.randint(1, 6))]
        simulate(plan, images, order, group, sms, ctas_per_sm, 6, ahead, rng)

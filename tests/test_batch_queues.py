"""The batched Richardson-Lucy run's queues (iane_gb300/csrc/rl_batch_kernel.cu, order "by
width"), restated in Python: one queue per PSF width, each CTA starting on the queue of its SM
and moving to the fullest other queue when its own is empty. A discrete-event simulation with
random durations checks that every item is done exactly once, that an item of phase p starts
only after its image has completed phase p - 1, and that the run never stalls."""
from __future__ import annotations

import random

import pytest


def run(classes, phases, ctas, seed):
    """classes: per queue, the tile counts of its images."""
    rng = random.Random(seed)
    images = [(c, i, n) for c, cls in enumerate(classes) for i, n in enumerate(cls)]
    queue = {c: [(i, t) for i, n in enumerate(cls) for t in range(n)] for c, cls in enumerate(classes)}
    head = {c: 0 for c in queue}
    done = {(c, i): 0 for c, i, _ in images}
    tiles = {(c, i): n for c, i, n in images}
    left = lambda c: len(queue[c]) * phases - head[c]  # noqa: E731
    at = [rng.randrange(len(classes)) for _ in range(ctas)]  # each CTA's queue
    held, busy, now, finished = [None] * ctas, [0.0] * ctas, 0.0, []
    closed = [False] * ctas
    for _ in range(100000):
        moved = False
        for k in range(ctas):
            if held[k] is not None and busy[k] and busy[k] <= now:
                c, p, i, t = held[k]
                done[c, i] += 1
                finished.append(held[k])
                held[k], busy[k], moved = None, 0.0, True
            if held[k] is None and not closed[k]:
                if left(at[k]) <= 0:
                    best = max(range(len(classes)), key=left)
                    if left(best) <= 0:
                        closed[k] = True
                        continue
                    at[k] = best
                c = at[k]
                p, e = divmod(head[c], len(queue[c]))
                head[c] += 1
                held[k], moved = (c, p, *queue[c][e]), True
            if held[k] is not None and not busy[k]:
                c, p, i, t = held[k]
                if done[c, i] >= p * tiles[c, i]:
                    assert done[c, i] < (p + 1) * tiles[c, i]  # no tile of the next phase was done
                    busy[k], moved = now + rng.uniform(0.5, 3.0), True
        if len(finished) == phases * sum(tiles.values()):
            assert len(set(finished)) == len(finished)
            return
        running = [b for b in busy if b]
        assert moved or running, "stalled"
        if not moved:
            now = min(running)
    raise AssertionError("did not end")


@pytest.mark.parametrize("ctas", [1, 2, 7, 40, 200])
@pytest.mark.parametrize("classes", [[[3]], [[1, 5, 2], [4]], [[2, 2], [9], [1, 1, 1], [6, 3]]])
def test_queues_order_every_phase_and_end(classes, ctas):
    for seed in range(3):
        run(classes, 6, ctas, seed)

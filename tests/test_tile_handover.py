"""Hand-over of accumulators from the watcher warp to the epilogue warps, in every interleaving of a small CTA (CPU).

A named barrier of as many arrivals as there are epilogue warps, plus the watcher's, releases the epilogue warps for a tile;
any wait of the watcher may run out.  The decisions are the kernels' own (csrc/tile_handover.cuh, compiled for the host);
the protocol around them is explored to the end, and every path has to end with all warps gone.
"""

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "dist_moe_b200" / "csrc"
WARPS, TILES = 2, 6

HARNESS = """
#include "tile_handover.cuh"
extern "C" int barrier(int it) { return dm::handover_barrier(it) - 1; }
extern "C" int none() { return dm::kNoBadTile; }
extern "C" int report(int* first_bad, int it, int came) { return dm::handover_report(first_bad, it, came != 0); }
extern "C" unsigned last_parity(int stage, unsigned phase, int s) { return dm::ring_last_parity(dm::ring_stop(stage, phase), s); }
extern "C" int good(const int* first_bad, int it) { return dm::handover_good(first_bad, it); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    folder = tmp_path_factory.mktemp("tile_handover")
    (folder / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-x", "c++", str(folder / "harness.cpp"), f"-I{CSRC}",
                    "-o", str(folder / "harness.so")], check=True)
    return ctypes.CDLL(str(folder / "harness.so"))


class Recorded:
    """The kernels' rule.  ``keep_arriving``: the watcher goes on arriving after the first bad tile; ``barriers``: that many
    take turns."""

    def __init__(self, lib, keep_arriving=False, barriers=None):
        self.lib, self.keep_arriving = lib, keep_arriving
        self.barrier = (lambda it: it % barriers) if barriers else lib.barrier

    def start(self):
        return self.lib.none()

    def watch(self, note, it, came):
        word = ctypes.c_int(note)
        if came or note == self.lib.none():
            went_on = bool(self.lib.report(ctypes.byref(word), it, int(came)))
            assert went_on == came
        return word.value, came or self.keep_arriving

    def good(self, note, it):
        return bool(self.lib.good(ctypes.byref(ctypes.c_int(note)), it))

    def disturb(self, note):
        return note


class Flag:
    """Every epilogue warp reads the flag that any role raises when it gives up; the watcher arrives for every tile."""

    def __init__(self, lib):
        self.barrier = lib.barrier

    def start(self):
        return 0

    def watch(self, note, it, came):
        return (note if came else 1), True

    def good(self, note, it):
        return note == 0

    def disturb(self, note):
        return 1


def stuck_paths(rule):
    """Number of reachable states that nothing leads out of although a warp is still there."""
    # state: note, watcher (tile, gave up), per warp (tile, step), arrivals at the barriers
    # steps of an epilogue warp: 0 reaches the barrier, 1 waits there, 2 decides, 3 stores and hands back, 9 gone
    first = (rule.start(), (0, False), ((0, 0),) * WARPS, (0,) * 4)
    todo, seen, stuck = [first], {first}, 0
    while todo:
        note, (wt, gave_up), warps, bars = state = todo.pop()
        after = []

        def arrive(warps, bars, b):
            n = bars[b] + 1
            if n == WARPS + 1:  # complete: released, counting from zero again
                warps = tuple((t, 2) if s == 1 and rule.barrier(t) == b else (t, s) for t, s in warps)
                n = 0
            return warps, tuple(n if i == b else v for i, v in enumerate(bars))

        if wt < TILES:
            handed_back = all(t > wt - 2 or s == 9 for t, s in warps) or wt < 2
            for came in ([True] if handed_back and not gave_up else []) + [False]:
                noted, go_on = rule.watch(note, wt, came)
                w, b = arrive(warps, bars, rule.barrier(wt))
                after.append((noted, ((wt + 1) if go_on else TILES, gave_up or not came), w, b))
        if rule.disturb(note) != note:
            after.append((rule.disturb(note), (wt, gave_up), warps, bars))
        for i, (t, s) in enumerate(warps):
            def put(t2, s2):
                return tuple((t2, s2) if j == i else v for j, v in enumerate(warps))
            if s == 0:
                if t == TILES:
                    after.append((note, (wt, gave_up), put(t, 9), bars))
                else:
                    w, b = arrive(put(t, 1), bars, rule.barrier(t))
                    after.append((note, (wt, gave_up), w, b))
            elif s == 2:
                after.append((note, (wt, gave_up), put(t, 3 if rule.good(note, t) else 9), bars))
            elif s == 3:
                after.append((note, (wt, gave_up), put(t + 1, 0), bars))
        after = [a for a in after if a != state]
        if not after and any(s != 9 for _, s in warps):
            stuck += 1
        for a in after:
            if a not in seen:
                seen.add(a)
                todo.append(a)
    return stuck


def test_every_warp_leaves_whatever_runs_out(lib):
    assert stuck_paths(Recorded(lib)) == 0


def test_what_the_rule_is_for(lib):
    """Warps that decide by a flag for themselves, a watcher that goes on arriving, and two barriers in turn, each leave a
    warp waiting alone."""
    assert stuck_paths(Flag(lib)) > 0
    assert stuck_paths(Recorded(lib, keep_arriving=True)) > 0
    assert stuck_paths(Recorded(lib, barriers=2)) > 0


def test_the_last_use_of_every_stage_is_what_is_waited_for(lib):
    """An mbarrier reports the parity of the phase before its current one as complete.  With every use of a role complete, the
    wait for its last use of each stage returns; with one use outstanding, the wait for that stage does not."""
    complete = lambda phases, parity: (phases - 1) & 1 == parity  # noqa: E731  (a fresh barrier: parity 1)
    rng = random.Random(5)
    for _ in range(300):
        stages, uses = rng.randint(1, 10), rng.randint(0, 45)
        stage, phase, done = 0, 0, [0] * stages
        for _ in range(uses):
            done[stage] += 1
            stage += 1
            if stage == stages:
                stage, phase = 0, phase ^ 1
        parity = [lib.last_parity(stage, phase, s) for s in range(stages)]
        assert all(complete(done[s], parity[s]) for s in range(stages))
        for back in range(min(uses, stages)):  # the latest uses may still be in flight
            s = (stage - 1 - back) % stages
            assert not complete(done[s] - 1, parity[s])

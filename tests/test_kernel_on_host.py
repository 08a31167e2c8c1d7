"""The search kernel's own code, run on the host.

Every thread of a launch is a fiber (tests/kernel_host/lanes.cpp): all 32 lanes
of a warp have to come to the same warp operation, warps run in a random order,
blocks stall for random times.  So the three kinds of team -- one block, a
cluster, a ring with its two independent hand-offs -- meet under many
interleavings, small enough to end within seconds, and their costs have to equal
the oracle's.  Planted mistakes in the ring's arithmetic have to be found."""
import os
import subprocess

import numpy as np
import pytest

import kernel_host

BLOCK, CLUSTER, RING = 0, 1, 2
STATUS = {"OK": 0, "NO_PATH": 1, "BUDGET": 2, "HEAP_FULL": 4, "TABLE_FULL": 5}


def _build(dst, edit=lambda name, text: text):
    kernel_host.rewrite(str(dst), "lanes.h", edit)
    exe = os.path.join(str(dst), "search")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "search_main.cpp", "lanes.cpp", "-o", exe], cwd=str(dst),
                   check=True)
    return exe


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("kernel"))


def _run(exe, inst, team, blocks, warps, ew, seed=1, wide=(0, 0), buckets=0, delta=0, slice=0, snodes=7, table_log2=16,
         cap=256, max_exp=0, max_iter=0):
    head, weights = inst
    cfg = (team, blocks, warps, ew, *wide, buckets, delta, slice, snodes, table_log2, cap, max_exp, max_iter, seed)
    text = " ".join(str(int(x)) for x in (*head, *cfg, *weights))
    r = subprocess.run([exe], input=text, capture_output=True, text=True, timeout=300)
    if r.returncode:
        return {"failed": r.returncode, "said": r.stdout[-200:]}
    v = [int(x) for x in r.stdout.split()]
    return dict(zip(("status", "cost", "iterations", "expansions", "stale", "generated", "pushes", "used", "launches"), v))


def _grid(gastar, oracle, w, h, seed, density=0.2):
    wts = gastar.gen_grid(w, h, seed, density)
    cost = oracle.grid_astar(wts, (0, 0), (w - 1, h - 1), path=False)[0].cost
    minw = int(wts[wts > 0].min())
    f0 = (max(w, h) - 1) * minw
    return ((3, w, h, 0, 0, w * h - 1, 0, minw, f0, 0), wts.reshape(-1).tolist()), cost


def _board(gastar, oracle, n, seed, walk):
    s, g = gastar.gen_sliding(n, seed, walk, walk)
    cost = oracle.sliding_astar(n, s, g, path=False)[0].cost
    bits = 4 if n < 5 else 5
    at = {int(t): i for i, t in enumerate(g)}
    f0 = sum(abs(i // n - at[int(t)] // n) + abs(i % n - at[int(t)] % n) for i, t in enumerate(s) if t)
    key = lambda b: sum(int(t) << (bits * i) for i, t in enumerate(b))
    lo = (1 << 64) - 1
    head = (n - 3, 0, 0, key(s) & lo, key(s) >> 64, key(g) & lo, key(g) >> 64, 0, f0, 0)
    return (head, []), cost


SHAPES = [(BLOCK, 1, 1), (BLOCK, 1, 3), (CLUSTER, 2, 2), (CLUSTER, 3, 1), (RING, 2, 2), (RING, 3, 1), (RING, 5, 2)]


@pytest.mark.parametrize("team,blocks,warps", SHAPES)
@pytest.mark.parametrize("slice", [0, 5])
def test_costs_under_random_interleavings(search, gastar, oracle, team, blocks, warps, slice):
    grid, gc = _grid(gastar, oracle, 31, 26, 3)
    b3, c3 = _board(gastar, oracle, 3, 7, 24)
    b4, c4 = _board(gastar, oracle, 4, 8, 22)
    b5, c5 = _board(gastar, oracle, 5, 9, 14)
    for inst, cost, ew, buckets, delta in ((grid, gc, 4, 0, 0), (grid, gc, 9, 1, 9), (b3, c3, 8, 0, 0), (b4, c4, 3, 1, 0),
                                           (b5, c5, 17, 0, 0)):
        r = _run(search, inst, team, blocks, warps, ew, seed=blocks + ew, buckets=buckets, delta=delta, slice=slice)
        assert r.get("status") == STATUS["OK"] and r["cost"] == cost, r
        assert (r["launches"] > 1) == (slice > 0)


@pytest.mark.parametrize("team", [CLUSTER, RING])
def test_widened_searches(search, gastar, oracle, team):
    for seed in range(4):
        inst, cost = _board(gastar, oracle, 4, 20 + seed, 26)
        r = _run(search, inst, team, 3, 2, 2, seed=seed, wide=(8, 4))
        assert r.get("status") == STATUS["OK"] and r["cost"] == cost, r


@pytest.mark.parametrize("team,blocks,warps", [(BLOCK, 1, 2), (CLUSTER, 3, 1), (RING, 3, 2)])
def test_searches_that_end_early(search, gastar, oracle, team, blocks, warps):
    inst, _ = _board(gastar, oracle, 4, 31, 40)
    assert _run(search, inst, team, blocks, warps, 4, max_iter=6)["status"] == STATUS["BUDGET"]
    assert _run(search, inst, team, blocks, warps, 4, max_exp=40)["status"] == STATUS["BUDGET"]
    assert _run(search, inst, team, blocks, warps, 4, table_log2=6)["status"] == STATUS["TABLE_FULL"]
    assert _run(search, inst, team, blocks, warps, 8, cap=14, table_log2=17)["status"] in (STATUS["HEAP_FULL"],
                                                                                          STATUS["OK"])
    wall = np.zeros((9, 9), dtype=np.uint8)
    wall[0, 0] = wall[8, 8] = 1
    inst = ((3, 9, 9, 0, 0, 80, 0, 1, 8, 0), wall.reshape(-1).tolist())
    assert _run(search, inst, team, blocks, warps, 4)["status"] == STATUS["NO_PATH"]


PLANTED = {
    "a stage ring one buffer short": ("engine_types.h", "constexpr uint32_t kStageRing = 4;",
                                      "constexpr uint32_t kStageRing = 3;"),
    "a cut cleared one iteration early": ("search.cuh", "cuts + (it - 2 * kCutLag - 2) % kCuts",
                                                       "cuts + (it - 2 * kCutLag - 1) % kCuts"),
    "a region published before it is complete": ("search.cuh", "(it + 1) << 32) | mine);",
                                                 "(it + 1) << 32) | (mine ? mine - 1 : 0));"),
}


@pytest.mark.parametrize("mistake", sorted(PLANTED))
def test_planted_mistakes_are_found(tmp_path, gastar, oracle, mistake):
    file, old, new = PLANTED[mistake]

    def plant(name, text):
        if name == "engine_types.h":
            text = text.replace("static_assert(kStageRing", "static_assert(true || kStageRing")
        if name == file:
            assert text.count(old) == 1
            text = text.replace(old, new)
        return text

    exe = _build(tmp_path, plant)
    for seed in range(12):
        inst, cost = _grid(gastar, oracle, 31, 26, 40 + seed)
        r = _run(exe, inst, RING, 5, 2, 4, seed=seed)
        if r.get("status") != STATUS["OK"] or r["cost"] != cost:
            return
    pytest.fail("not found")

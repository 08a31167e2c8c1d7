"""Measured cases: what a user has this engine do, through `cuda_a_star_gb300`.

Plain solves of one instance (sliding puzzles 3x3 to 5x5 and weighted grids,
host or device weights, with and without a pop window), batches of many
instances (one call from host buffers to results, and device-resident re-runs)
and bursts of mixed requests on the server.  Inputs are the repository's own
benchmark and test workloads: puzzles scrambled from the goal by non-reversing
random walks, grids of weights 1-9 with 10-30 % obstacles and a guaranteed
corridor.

Several optimal paths usually tie, and which one a parallel search returns
differs from run to run.  So a pass returns what is the same for all of them:
the cost, the endpoints, and per step what a path has to satisfy (two cells of
the board change; a grid path's weights add up to its cost).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import cuda_a_star_gb300 as g

# One engine per process, as a program keeps it; one server beside it.
_ENGINE = None
_SERVER = None
_SERVER_BUDGET = 48 << 30


def _engine():
    global _ENGINE
    if _ENGINE is None:
        _ENGINE = g.Engine(0)
    return _ENGINE


def _server():
    global _SERVER
    if _SERVER is None:
        _SERVER = _engine().server(budget_bytes=_SERVER_BUDGET)
    return _SERVER


# ---- the cases ----

def listed():
    return [
        # One 8-puzzle at the default 4096 queues: the smallest call, all latency.
        {"name": "p8", "what": "sliding", "n": 3, "queues": 4096, "table_log2": 0,
         "walk_min": 60, "walk_max": 60, "count": 1},
        # Ordinary 15-puzzles with the default configuration.
        {"name": "p15_default", "what": "sliding", "n": 4, "queues": 4096, "table_log2": 0,
         "walk_min": 20, "walk_max": 80, "count": 8},
        # The headline benchmark's puzzles and configuration, a part of its 64.
        {"name": "p15_wide", "what": "sliding", "n": 4, "queues": 16384, "table_log2": 30,
         "walk_min": 40, "walk_max": 80, "count": 16},
        # 24-puzzles (128-bit keys) as the served mix has them.
        {"name": "p24", "what": "sliding", "n": 5, "queues": 4096, "table_log2": 0,
         "walk_min": 20, "walk_max": 40, "count": 8},
        # A small grid with the default configuration (the reference's range).
        {"name": "grid_200x150", "what": "grid", "w": 200, "h": 150, "density": 0.2, "queues": 4096,
         "delta": 0, "heuristic": 0, "device": False, "inside": False},
        # A ragged grid searched without a heuristic (Dijkstra), inner endpoints.
        {"name": "grid_517x389_zero", "what": "grid", "w": 517, "h": 389, "density": 0.25,
         "queues": 4096, "delta": 0, "heuristic": 2, "device": False, "inside": True},
        # A map that already is on the device, cost only.
        {"name": "grid_1021_device", "what": "grid", "w": 1021, "h": 1021, "density": 0.2,
         "queues": 16384, "delta": 72, "heuristic": 0, "device": True, "inside": False},
        # The benchmark's large grid with its pop window.
        {"name": "grid_4096", "what": "grid", "w": 4096, "h": 4096, "density": 0.2, "queues": 16384,
         "delta": 72, "heuristic": 0, "device": False, "inside": False},
        # Many small puzzles in one call.
        {"name": "batch_p8", "what": "batch", "p8": 512, "p15": 0, "p24": 0, "grids": 0,
         "side_min": 0, "side_max": 0, "walk_max": 60, "again": False},
        # A mixed batch in one call: upload, search, paths back.
        {"name": "batch_mixed", "what": "batch", "p8": 0, "p15": 64, "p24": 0, "grids": 64,
         "side_min": 256, "side_max": 2048, "walk_max": 80, "again": False},
        # A resident batch of grids solved again (replanning on the same maps).
        {"name": "batch_grids_again", "what": "batch", "p8": 0, "p15": 0, "p24": 0, "grids": 152,
         "side_min": 256, "side_max": 1024, "walk_max": 0, "again": True},
        # A burst of mixed requests on the server, drained.
        {"name": "served_burst", "what": "served", "p8": 12, "p15": 12, "p24": 12, "grids": 12,
         "side_min": 512, "side_max": 3072, "walk_max": 80},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    what = rng.choice(["sliding", "sliding", "grid", "grid", "grid", "batch", "batch", "served"])
    if what == "sliding":
        n = rng.choice([3, 4, 4, 5])
        hi = {3: 70, 4: 80, 5: 40}[n]
        lo = rng.randint(16, hi)
        return {"what": what, "n": n, "queues": rng.choice([256, 1024, 4096, 8192, 16384, 3000]),
                "table_log2": rng.choice([0, 0, 24]), "walk_min": lo, "walk_max": rng.randint(lo, hi),
                "count": rng.randint(1, 12)}
    if what == "grid":
        w = _log_int(rng, 48, 3000)
        h = max(33, min(3000, int(w * rng.uniform(0.5, 1.6))))
        wide = rng.random() < 0.6
        return {"what": what, "w": w, "h": h, "density": round(rng.uniform(0.1, 0.3), 3),
                "queues": rng.choice([4096, 16384]) if w * h < 1 << 20 or wide else 16384,
                "delta": rng.choice([18, 36, 72]) if wide or w * h > 1 << 20 else 0,
                "heuristic": rng.choice([0, 0, 0, 2]) if w * h < 1 << 20 else 0,
                "device": rng.random() < 0.3, "inside": rng.random() < 0.5}
    if what == "batch":
        lo = rng.randint(64, 512)
        return {"what": what, "p8": rng.choice([0, rng.randint(1, 200)]), "p15": rng.randint(1, 64),
                "p24": rng.choice([0, rng.randint(1, 16)]), "grids": _log_int(rng, 2, 64),
                "side_min": lo, "side_max": rng.randint(lo, 1600), "walk_max": rng.randint(30, 80),
                "again": rng.random() < 0.5}
    lo = rng.randint(128, 1024)
    return {"what": what, "p8": rng.randint(1, 16), "p15": rng.randint(1, 16), "p24": rng.randint(1, 16),
            "grids": rng.randint(1, 12), "side_min": lo, "side_max": rng.randint(lo, 2800),
            "walk_max": rng.randint(40, 80)}


# ---- inputs ----

def _scramble(n, steps, rng):
    """A board `steps` non-reversing blank moves away from 0..n*n-1."""
    b = list(range(n * n))
    blank, last = 0, None
    while steps:
        dr, dc = rng.choice(((1, 0), (-1, 0), (0, 1), (0, -1)))
        r, c = blank // n + dr, blank % n + dc
        if not (0 <= r < n and 0 <= c < n) or (last is not None and (dr, dc) == (-last[0], -last[1])):
            continue
        q = r * n + c
        b[blank], b[q] = b[q], 0
        blank, last = q, (dr, dc)
        steps -= 1
    return np.array(b, dtype=np.uint8), np.arange(n * n, dtype=np.uint8)


def _grid(w, h, density, inside, seed):
    """Weights 1-9, obstacles (0) with the given density, and a passable
    staircase corridor between the corners; on the GPU.  Endpoints: the
    corners, or two cells on the corridor."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randint(1, 10, (h, w), dtype=torch.uint8, device="cuda", generator=gen)
    keep = torch.rand((h, w), device="cuda", generator=gen) >= density
    steps = torch.zeros(w + h - 2, dtype=torch.int64, device="cuda")
    steps[: w - 1] = 1
    steps = steps[torch.randperm(w + h - 2, device="cuda", generator=gen)]
    zero = torch.zeros(1, dtype=torch.int64, device="cuda")
    x = torch.cat([zero, torch.cumsum(steps, 0)])
    y = torch.cat([zero, torch.cumsum(1 - steps, 0)])
    keep[y, x] = True
    a = a * keep
    i, j = (len(x) // 8, len(x) - 1 - len(x) // 8) if inside else (0, len(x) - 1)
    at = torch.stack([x[[i, j]], y[[i, j]]], 1).cpu().numpy()
    return a, (int(at[0, 0]), int(at[0, 1])), (int(at[1, 0]), int(at[1, 1]))


def _mix(case, seed):
    """The instances of a batch or a burst, in a shuffled order."""
    rng = random.Random(seed * 7919 + 17)
    out = []
    for n, key, lo, hi in ((3, "p8", 60, 60), (4, "p15", 20, case["walk_max"]), (5, "p24", 20, 40)):
        out += [("s", *_scramble(n, rng.randint(lo, max(lo, hi)), rng)) for _ in range(case[key])]
    for _ in range(case["grids"]):
        side = rng.randint(case["side_min"], case["side_max"])
        a, st, gl = _grid(side, side, rng.uniform(0.1, 0.3), False, rng.randrange(1 << 40))
        out.append(("g", a.cpu().numpy(), st, gl))
    rng.shuffle(out)
    return out


def _single_boards(case, seed):
    rng = random.Random(seed * 7919 + 17)
    return [_scramble(case["n"], rng.randint(case["walk_min"], case["walk_max"]), rng)
            for _ in range(case["count"])]


def _batch(eng, insts):
    """A batch of these instances, in the default shape; 24-puzzles' larger
    entries need blocks of 8 warps."""
    wide = any(p[0] == "s" and len(p[1]) == 25 for p in insts)
    batch = eng.batch(warps_per_block=8) if wide else eng.batch()
    for p in insts:
        if p[0] == "s":
            batch.add_sliding(p[1], p[2])
        else:
            batch.add_grid(p[1], p[2], p[3])
    return batch


def prepare(case, seed):
    eng = _engine()
    what = case["what"]
    if what == "sliding":
        cfg = g.make_config(num_queues=case["queues"], table_log2=case["table_log2"])
        return {"what": what, "eng": eng, "boards": _single_boards(case, seed), "n": case["n"], "cfg": cfg,
                "most": case["walk_max"]}
    if what == "grid":
        a, st, gl = _grid(case["w"], case["h"], case["density"], case["inside"], seed)
        cfg = g.make_config(num_queues=case["queues"], delta=case["delta"], heuristic=case["heuristic"])
        if case["device"]:
            torch.cuda.synchronize()
            return {"what": "grid_device", "eng": eng, "w": a, "start": st, "goal": gl, "cfg": cfg}
        return {"what": what, "eng": eng, "w": a.cpu().numpy(), "start": st, "goal": gl, "cfg": cfg}
    insts = _mix(case, seed)
    state = {"what": what, "eng": eng, "insts": insts}
    if what == "batch" and case["again"]:
        state["batch"] = _batch(eng, insts)
        state["batch"].run()
    if what == "served":
        state["server"] = _server()
    return state


# ---- one pass ----

def _board_steps(p, most):
    """Cells that change in each step of a board path (0 past its end)."""
    steps = np.zeros(most, dtype=np.int64)
    steps[: len(p) - 1] = (p[1:] != p[:-1]).sum(1)
    return steps


def _results(insts, results):
    status = np.array([r.status for r in results])
    cost = np.array([r.cost for r in results])
    length, total = [], []
    for p, r in zip(insts, results):
        if p[0] == "s":
            length.append(len(r.path))
        else:
            total.append(int(p[1].reshape(-1)[r.path[1:]].sum(dtype=np.int64)))
    return {"status": status, "cost": cost, "board_path_states": np.array(length, dtype=np.int64),
            "grid_path_cost": np.array(total, dtype=np.int64)}


def run(state):
    eng, what = state["eng"], state["what"]
    if what == "sliding":
        rs = [eng.solve_sliding(s, t, state["n"], config=state["cfg"], path_cap=1024) for s, t in state["boards"]]
        return {"status": np.array([r.status for r in rs]), "cost": np.array([r.cost for r in rs]),
                "changed": np.stack([_board_steps(r.path, state["most"]) for r in rs]),
                "first": np.stack([r.path[0] for r in rs]), "last": np.stack([r.path[-1] for r in rs])}
    if what == "grid":
        w = state["w"]
        r = eng.solve_grid(w, state["start"], state["goal"], config=state["cfg"])
        return {"status": r.status, "cost": r.cost, "path_cost": int(w.reshape(-1)[r.path[1:]].sum(dtype=np.int64)),
                "ends": r.path[[0, -1]].astype(np.int64)}
    if what == "grid_device":
        w = state["w"]
        r = eng.solve_grid_device(w.data_ptr(), w.shape[1], w.shape[0], state["start"], state["goal"],
                                  config=state["cfg"])
        return {"status": r.status, "cost": r.cost}
    insts = state["insts"]
    if what == "batch":
        b = state.get("batch")
        if b is not None:
            b.rerun()
            return _results(insts, [b.result(i) for i in range(len(insts))])
        b = _batch(eng, insts)
        b.run()
        out = _results(insts, [b.result(i) for i in range(len(insts))])
        b.close()
        return out
    srv = state["server"]
    ids = [srv.submit_sliding(p[1], p[2]) if p[0] == "s" else srv.submit_grid(p[1], p[2], p[3]) for p in insts]
    done = srv.drain(ids)
    for i in ids:
        srv.release(i)
    return _results(insts, [done[i] for i in ids])


# ---- what a pass cannot do without ----

def work(case):
    """Inputs read once and results written once.  A search that proves a cost
    also touches every state with f below it; that count depends on the
    instance and is left out."""
    if case["what"] == "sliding":
        cells = case["n"] ** 2
        return {"bytes": case["count"] * cells * (2 + case["walk_min"]), "flops": 0}
    if case["what"] == "grid":
        return {"bytes": case["w"] * case["h"] + 4 * max(case["w"], case["h"]), "flops": 0}
    side = (case["side_min"] + case["side_max"]) / 2
    return {"bytes": case["p8"] * 200 + case["p15"] * 600 + case["p24"] * 800 +
            case["grids"] * (side * side + 4 * side), "flops": 0}


# ---- the same, by other means ----

def _grid_cost(w, start, goal):
    """Least cost by buckets of equal distance (Dial), vectorised per bucket."""
    h, wd = w.shape
    pad = np.zeros((h + 2, wd + 2), dtype=np.int64)
    pad[1:-1, 1:-1] = w
    cost = pad.reshape(-1)
    row = wd + 2
    dist = np.full(cost.shape, np.iinfo(np.int64).max, dtype=np.int64)
    s, t = (start[1] + 1) * row + start[0] + 1, (goal[1] + 1) * row + goal[0] + 1
    dist[s] = 0
    buckets = [[] for _ in range(10)]
    buckets[0].append(np.array([s]))
    offs = np.array([-row - 1, -row, -row + 1, -1, 1, row - 1, row, row + 1])
    d, empty = 0, 0
    while empty < 10:
        todo, buckets[d % 10] = buckets[d % 10], []
        cells = np.unique(np.concatenate(todo)) if todo else np.zeros(0, dtype=np.int64)
        cells = cells[dist[cells] == d]
        if len(cells) == 0:
            d, empty = d + 1, empty + 1
            continue
        empty = 0
        if dist[t] == d:
            return d
        nb = (cells[:, None] + offs).reshape(-1)
        nb = nb[cost[nb] > 0]
        nd = d + cost[nb]
        better = nd < dist[nb]
        nb, nd = nb[better], nd[better]
        np.minimum.at(dist, nb, nd)
        for k in range(1, 10):
            at = nb[(nd == d + k) & (dist[nb] == nd)]
            if len(at):
                buckets[(d + k) % 10].append(at)
        d += 1
    return None


def _board_cost8(start):
    """Breadth-first distance of a 3x3 board from 0..8."""
    goal, start = tuple(range(9)), tuple(int(v) for v in start)
    seen, edge, d = {goal}, [goal], 0
    while edge:
        if start in seen:
            return d
        nxt = []
        for b in edge:
            z = b.index(0)
            for dr, dc in ((1, 0), (-1, 0), (0, 1), (0, -1)):
                r, c = z // 3 + dr, z % 3 + dc
                if 0 <= r < 3 and 0 <= c < 3:
                    m = list(b)
                    q = r * 3 + c
                    m[z], m[q] = m[q], 0
                    m = tuple(m)
                    if m not in seen:
                        seen.add(m)
                        nxt.append(m)
        edge, d = nxt, d + 1
    return None


def exact(case, seed):
    if case["what"] == "sliding" and case["n"] == 3:
        boards = _single_boards(case, seed)
        cost = np.array([_board_cost8(s) for s, _ in boards])
        return {"status": np.zeros(len(boards), dtype=np.int64), "cost": cost,
                "changed": 2 * (np.arange(case["walk_max"]) < cost[:, None]).astype(np.int64), "first": np.stack([s for s, _ in boards]),
                "last": np.stack([t for _, t in boards])}
    if case["what"] == "grid" and case["w"] * case["h"] <= 1 << 21:
        a, st, gl = _grid(case["w"], case["h"], case["density"], case["inside"], seed)
        c = _grid_cost(a.cpu().numpy(), st, gl)
        if case["device"]:
            return {"status": 0, "cost": c}
        return {"status": 0, "cost": c, "path_cost": c,
                "ends": np.array([st[1] * case["w"] + st[0], gl[1] * case["w"] + gl[0]])}
    return None

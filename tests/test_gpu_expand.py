"""Expansion rounds of the search kernel: a warp expands its popped entries a
few per round (four grid cells or eight boards), so pop widths around a
round's and a batch of rounds' edges, one block and several, heaps and
buckets.  Costs are whole numbers and equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WIDTHS = [1, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32]


@pytest.mark.parametrize("blocks", [1, 3])
@pytest.mark.parametrize("width", WIDTHS)
def test_pop_widths(engine, oracle, gastar, width, blocks):
    kw = dict(expansion_width=width, warps_per_block=2, num_queues=2 * width * blocks)
    for w, h, delta in ((7, 1, 0), (33, 20, 0), (61, 47, 9)):
        wts = gastar.gen_grid(w, h, 40 + w, 0.2)
        r = engine.solve_grid(wts, (0, 0), (w - 1, h - 1), delta=delta, **kw)
        o, _ = oracle.grid_astar(wts, (0, 0), (w - 1, h - 1), path=False)
        assert r.status_name == "OK" and r.cost == o.cost
        assert oracle.grid_validate(wts, (0, 0), (w - 1, h - 1), r.path) == (True, r.cost)
    for n, walk in ((3, (20, 30)), (4, (16, 24)), (5, (10, 16))):
        s, g = gastar.gen_sliding(n, 70 + n, *walk)
        r = engine.solve_sliding(s, g, n, **kw)
        o, _ = oracle.sliding_astar(n, s, g, path=False)
        assert r.status_name == "OK" and r.cost == o.cost
        assert oracle.sliding_validate(n, s, g, r.path) == (True, r.cost)


@pytest.mark.parametrize("warps", [1, 5, 8, 9, 16])
def test_block_shapes_in_a_batch(engine, oracle, gastar, warps):
    """One-block teams of every warp count class, with and without buckets."""
    for open_list in (0, 1):
        b = engine.batch(warps_per_block=warps, expansion_width=17, open_list=open_list)
        cases = []
        for i in range(4):
            side = 30 + 17 * i
            wts = gastar.gen_grid(side, side + 3, 90 + i, 0.25)
            b.add_grid(wts, (0, 0), (side - 1, side + 2))
            cases.append(oracle.grid_astar(wts, (0, 0), (side - 1, side + 2), path=False)[0].cost)
            s, g = gastar.gen_sliding(3 + i % 2, 95 + i, 20, 30)
            b.add_sliding(s, g)
            cases.append(oracle.sliding_astar(3 + i % 2, s, g, path=False)[0].cost)
        b.run()
        assert [b.result(i, path=False).cost for i in range(len(b))] == cases
        b.rerun()
        assert [b.result(i, path=False).cost for i in range(len(b))] == cases
        b.close()


@pytest.mark.parametrize("blocks,warps", [(2, 1), (2, 8), (3, 3), (7, 2), (15, 8), (16, 1), (16, 8), (17, 8)])
def test_cluster_teams(engine, oracle, gastar, blocks, warps):
    """Clusters of every size class (17 blocks: a ring team), heaps and
    buckets, a budget that ends the search early, then a normal solve."""
    for open_list in (0, 1):
        kw = dict(expansion_width=4, warps_per_block=warps, num_queues=4 * warps * blocks, open_list=open_list)
        for w, h, delta in ((5, 3, 0), (83, 64, 0), (83, 64, 12)):
            wts = gastar.gen_grid(w, h, 140 + w, 0.2)
            r = engine.solve_grid(wts, (0, 0), (w - 1, h - 1), delta=delta, **kw)
            o, _ = oracle.grid_astar(wts, (0, 0), (w - 1, h - 1), path=False)
            assert r.status_name == "OK" and r.cost == o.cost
            assert oracle.grid_validate(wts, (0, 0), (w - 1, h - 1), r.path) == (True, r.cost)
            assert r.expansions > 0 and r.generated >= r.pushes > 0
        for n, walk in ((3, (24, 30)), (4, (20, 30)), (5, (12, 18))):
            s, g = gastar.gen_sliding(n, 170 + n, *walk)
            r = engine.solve_sliding(s, g, n, **kw)
            o, _ = oracle.sliding_astar(n, s, g, path=False)
            assert r.status_name == "OK" and r.cost == o.cost
            assert oracle.sliding_validate(n, s, g, r.path) == (True, r.cost)
        s, g = gastar.gen_sliding(4, 199, 60, 60)
        r = engine.solve_sliding(s, g, 4, max_iterations=3, **kw)
        assert r.status_name == "BUDGET" and r.iterations <= 6
        wall = np.zeros((9, 9), dtype=np.uint8)
        wall[0, 0] = wall[8, 8] = 1
        assert engine.solve_grid(wall, (0, 0), (8, 8), **kw).status_name == "NO_PATH"


def test_cluster_heap_overflow_is_regrown(engine, oracle, gastar):
    """A heap that fills in a cluster team loses entries: without regrow the
    status says so, with it the cost is right."""
    wts = gastar.gen_grid(220, 180, 77, 0.1)
    o, _ = oracle.grid_astar(wts, (0, 0), (219, 179), path=False)
    kw = dict(expansion_width=1, warps_per_block=1, num_queues=2, heap_entries=1, heuristic=2)
    r = engine.solve_grid(wts, (0, 0), (219, 179), **kw)
    assert r.status_name == "OK" and r.cost == o.cost


@pytest.mark.parametrize("team", [2, 3, 4, 8, 16, 17])
@pytest.mark.parametrize("instances", [2, 150])
def test_heavy_teams(engine, oracle, gastar, team, instances):
    """Heavy grids solved by clusters, or by ring teams where the clusters of
    all teams are not resident at once (many instances) or the size is not a
    cluster's (17): one launch of a batch, and a server whose searches are
    suspended every few iterations with part of their roots popped."""
    sides = [40 + (7 * i) % 23 for i in range(instances)]
    grids = [gastar.gen_grid(s, s + 2, 300 + i, 0.2) for i, s in enumerate(sides)]
    want = [oracle.grid_astar(w, (0, 0), (s - 1, s + 1), path=False)[0].cost for w, s in zip(grids, sides)]
    kw = dict(warps_per_block=2, expansion_width=3, heavy_team=team, heavy_cells=1000)
    b = engine.batch(**kw)
    for w, s in zip(grids, sides):
        b.add_grid(w, (0, 0), (s - 1, s + 1))
    b.run()
    assert [b.result(i, path=False).cost for i in range(instances)] == want
    b.close()
    srv = engine.server(slice_iters=16, budget_bytes=4 << 30, heavy_teams=min(instances, 8), **kw)
    ids = [srv.submit_grid(w, (0, 0), (s - 1, s + 1)) for w, s in zip(grids, sides)]
    got = srv.drain(ids)
    srv.close()
    assert [got[i].cost for i in ids] == want
    for i, w, s in zip(ids, grids, sides):
        assert oracle.grid_validate(w, (0, 0), (s - 1, s + 1), got[i].path) == (True, got[i].cost)

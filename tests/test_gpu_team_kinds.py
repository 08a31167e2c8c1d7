"""Which kind of team runs, and heaps that overflow in each kind.

A search whose start is its goal tells the kind: one block and a cluster test
the start's iteration in that iteration, a ring two iterations later."""
import pytest

pytestmark = pytest.mark.gpu

BLOCK_OR_CLUSTER, RING = 0, 2  # iterations of a search that starts at its goal

SHAPES = {"block": dict(num_queues=32), "cluster": dict(num_queues=64), "ring": dict(num_queues=17 * 32)}


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_heap_overflow(engine, oracle, gastar, shape):
    """One-warp blocks have 8128 entries per heap at least; a blind search at
    depth 18 holds half a million."""
    s, g = gastar.gen_sliding(4, 918, 18, 18)
    want = oracle.sliding_astar(4, s, g, path=False)[0].cost
    assert want == 18
    kw = dict(expansion_width=32, warps_per_block=1, heap_entries=8192, heuristic=gastar.H_ZERO, **SHAPES[shape])
    at_goal = engine.solve_sliding(g, g, 4, **kw)
    assert at_goal.cost == 0 and at_goal.iterations == (RING if shape == "ring" else BLOCK_OR_CLUSTER)
    r = engine.solve_sliding(s, g, 4, regrow=0, **kw)
    assert r.status_name == "HEAP_FULL" and r.attempts == 1
    r = engine.solve_sliding(s, g, 4, **kw)
    assert r.status_name == "OK" and r.cost == want and r.attempts > 1
    assert oracle.sliding_validate(4, s, g, r.path) == (True, want)


@pytest.mark.parametrize("team,count,warps,kind", [
    (2, 6, 2, BLOCK_OR_CLUSTER), (4, 12, 8, BLOCK_OR_CLUSTER), (8, 24, 2, BLOCK_OR_CLUSTER),
    (16, 48, 8, BLOCK_OR_CLUSTER),  # few blocks: clusters
    (3, 9, 2, RING), (17, 51, 2, RING),  # no cluster's size
    (16, 160, 16, RING),  # 152 blocks, one per SM, are no whole number of clusters
])
def test_heavy_teams_of_a_batch(engine, oracle, gastar, team, count, warps, kind):
    b = engine.batch(warps_per_block=warps, expansion_width=32, heavy_team=team, heavy_cells=1000)
    want = []
    for i in range(count):
        side = 40 + (7 * i) % 23 if i % 3 else 20 + i % 10  # every third on one block
        w = gastar.gen_grid(side, side + 2, 600 + i, 0.2)
        b.add_grid(w, (0, 0), (side - 1, side + 1))
        want.append(oracle.grid_astar(w, (0, 0), (side - 1, side + 1), path=False)[0].cost)
    w = gastar.gen_grid(50, 50, 9, 0.0)
    probe = b.add_grid(w, (7, 7), (7, 7))
    b.run()
    assert b.result(probe).cost == 0 and b.result(probe).iterations == kind
    assert [b.result(i, path=False).cost for i in range(count)] == want
    b.rerun()
    assert b.result(probe).iterations == kind
    assert [b.result(i, path=False).cost for i in range(count)] == want
    b.close()


def test_requests_go_from_clusters_to_rings_and_back(engine, oracle, gastar):
    """Two heavy grids, suspended every 16 iterations: alone in clusters, in
    rings while one-block requests fill the device, then in clusters again."""
    srv = engine.server(heavy_team=16, heavy_cells=10000, slice_iters=16, budget_bytes=6 << 30)
    want, grids = {}, {}

    def submit(side, seed):
        w = gastar.gen_grid(side, side, seed, 0.2)
        i = srv.submit_grid(w, (0, 0), (side - 1, side - 1))
        grids[i], want[i] = w, oracle.grid_astar(w, (0, 0), (side - 1, side - 1), path=False)[0].cost
        return i

    def kind_of_a_step():
        i = srv.submit_grid(gastar.gen_grid(120, 120, 9, 0.0), (7, 7), (7, 7))
        srv.step()
        return srv.poll(i).iterations

    heavy = [submit(700, 1), submit(690, 2)]
    assert kind_of_a_step() == BLOCK_OR_CLUSTER
    light = [submit(60 + i % 9, 10 + i) for i in range(140)]
    assert kind_of_a_step() == RING
    assert kind_of_a_step() == RING
    got = srv.drain(light)
    assert all(srv.poll(i) is None for i in heavy)  # still at work
    assert kind_of_a_step() == BLOCK_OR_CLUSTER
    got.update(srv.drain(heavy))
    srv.close()
    assert {i: got[i].cost for i in got} == want
    for i in heavy:
        h, w = grids[i].shape
        assert oracle.grid_validate(grids[i], (0, 0), (w - 1, h - 1), got[i].path) == (True, want[i])


@pytest.mark.parametrize("queues", [64, 512])
def test_clusters_widen(engine, oracle, gastar, queues):
    """A puzzle that is past 64 iterations on a cluster takes fewer of them with
    the automatic width than with that width fixed."""
    s, g = gastar.gen_sliding(4, 909, 40, 70)
    want = oracle.sliding_astar(4, s, g, path=False)[0].cost
    auto = engine.solve_sliding(s, g, 4, num_queues=queues)
    fixed = engine.solve_sliding(s, g, 4, num_queues=queues, expansion_width=4, warps_per_block=8)
    for r in (auto, fixed):
        assert r.status_name == "OK" and r.cost == want
        assert oracle.sliding_validate(4, s, g, r.path) == (True, want)
    assert fixed.iterations > 128 and auto.iterations < fixed.iterations

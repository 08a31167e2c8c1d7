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

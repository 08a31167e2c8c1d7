"""The blocks of a batch's launch stay within the caller's cap, whatever teams
its heavy instances run in: no more blocks than that are at work at any time of
the launch's schedule."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks,team", [(3, 2), (5, 4), (6, 4), (7, 3), (4, 2)])
def test_schedule_fits_the_block_cap(engine, oracle, gastar, blocks, team):
    sides = [400] + [250 + 3 * i for i in range(2 * blocks)]
    b = engine.batch(blocks=blocks, heavy_team=team, heavy_cells=400 * 400)
    want = []
    for i, s in enumerate(sides):
        w = gastar.gen_grid(s, s, 500 + i, 0.2)
        b.add_grid(w, (0, 0), (s - 1, s - 1))
        want.append(oracle.grid_astar(w, (0, 0), (s - 1, s - 1), path=False)[0].cost)
    b.run()
    assert [b.result(i, path=False).cost for i in range(len(b))] == want
    start, end = b.timeline()
    b.close()
    held = [team] + [1] * (len(sides) - 1)
    most = max(sum(h for h, s, e in zip(held, start, end) if s <= t < e) for t in start)
    assert most <= blocks

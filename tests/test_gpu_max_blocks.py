"""max_blocks: searches whose team the caller caps, down to one block, which
then stages its successors in shared memory.  Costs equal the oracle's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 2, 16, 17])
def test_capped_teams(engine, oracle, gastar, cap):
    for open_list in (0, 1):
        kw = dict(max_blocks=cap, open_list=open_list)
        for n, walk in ((3, (24, 30)), (4, (40, 50)), (5, (24, 30))):
            s, g = gastar.gen_sliding(n, 270 + n, *walk)
            r = engine.solve_sliding(s, g, n, **kw)
            o, _ = oracle.sliding_astar(n, s, g, path=False)
            assert r.status_name == "OK" and r.cost == o.cost
            assert oracle.sliding_validate(n, s, g, r.path) == (True, r.cost)
        for w, h in ((60, 41), (391, 363)):
            wts = gastar.gen_grid(w, h, 240 + w, 0.2)
            r = engine.solve_grid(wts, (0, 0), (w - 1, h - 1), **kw)
            o, _ = oracle.grid_astar(wts, (0, 0), (w - 1, h - 1), path=False)
            assert r.status_name == "OK" and r.cost == o.cost
            assert oracle.grid_validate(wts, (0, 0), (w - 1, h - 1), r.path) == (True, r.cost)
        for width, warps in ((32, 8), (32, 16), (5, 9)):  # fixed widths of a ring's
            s, g = gastar.gen_sliding(5, 281, 20, 26)
            if cap == 1 and open_list and width * warps == 512:
                # One block's two stage buffers, heaps and bucket scratch are
                # 228 KiB, more than a block has: refused, as for a Q that
                # needs one block only.
                for kq in (dict(num_queues=512, open_list=1), dict(num_queues=16384, **kw)):
                    with pytest.raises(gastar.GastarError):
                        engine.solve_sliding(s, g, 5, expansion_width=width, warps_per_block=warps, **kq)
                continue
            r = engine.solve_sliding(s, g, 5, num_queues=16384, expansion_width=width, warps_per_block=warps, **kw)
            o, _ = oracle.sliding_astar(5, s, g, path=False)
            assert r.status_name == "OK" and r.cost == o.cost

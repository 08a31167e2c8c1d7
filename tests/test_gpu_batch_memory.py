"""Batches of one context one after the other, side by side and after larger or
smaller ones: a destroyed batch's device memory serves the next one, and the
context's end gives it back."""
import pytest

pytestmark = pytest.mark.gpu


def _batch(eng, gastar, oracle, count, seed, **kw):
    b = eng.batch(**kw)
    want = []
    for i in range(count):
        s, g = gastar.gen_sliding(4, seed + i, 20, 34)
        b.add_sliding(s, g)
        want.append(oracle.sliding_astar(4, s, g, path=False)[0].cost)
        side = 25 + (seed + 7 * i) % 40
        w = gastar.gen_grid(side, side, seed + i, 0.2)
        b.add_grid(w, (0, 0), (side - 1, side - 1))
        want.append(oracle.grid_astar(w, (0, 0), (side - 1, side - 1), path=False)[0].cost)
    return b, want


def test_batches_in_a_row_and_side_by_side(gastar, oracle):
    import torch
    with gastar.Engine(0) as eng:
        eng.solve_grid(gastar.gen_grid(9, 9, 1, 0.0), (0, 0), (8, 8))
        for count, seed in ((3, 10), (9, 40), (2, 80), (9, 40)):
            b, want = _batch(eng, gastar, oracle, count, seed)
            b.run()
            assert [b.result(i, path=False).cost for i in range(len(b))] == want
            c, want_c = _batch(eng, gastar, oracle, 2, seed + 5)  # while b is alive
            c.run()
            b.rerun()
            assert [b.result(i, path=False).cost for i in range(len(b))] == want
            assert [c.result(i, path=False).cost for i in range(len(c))] == want_c
            b.close()
            c.rerun()
            assert [c.result(i, path=False).cost for i in range(len(c))] == want_c
            c.close()
        kept = torch.cuda.mem_get_info()[0]
        srv = eng.server(budget_bytes=1 << 30)  # takes its budget from all free memory
        srv.close()
        assert torch.cuda.mem_get_info()[0] > kept
        b, want = _batch(eng, gastar, oracle, 3, 10)
        b.run()
        assert [b.result(i, path=False).cost for i in range(len(b))] == want
        b.close()
        kept = torch.cuda.mem_get_info()[0]
    assert torch.cuda.mem_get_info()[0] > kept

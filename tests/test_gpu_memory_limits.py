"""Device memory at its limits: calls that run out of it report so, later calls
work, and nothing stays allocated once batches and contexts are closed."""
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20
SIDE = 65535


def _free():
    import torch
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _fill(leave):
    """Takes all but `leave` bytes of the device's free memory."""
    import torch
    return torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")


def _long_grids(eng, count):
    """Grids of one row: their path arenas (2 MiB each) are a large part of a
    batch's memory beside the partitions."""
    import numpy as np
    b = eng.batch()
    w = np.ones((1, SIDE), dtype=np.uint8)
    for i in range(count):
        b.add_grid(w, (10 * i, 0), (10 * i + 5, 0))
    return b


def _partitions(b, count):
    paths = count * 4 * (1 + SIDE) * 8
    return b.stats()["device_bytes"] - 256 * MIB - paths


def _solved(b):
    return all(b.result(i).cost == 5 and len(b.result(i).path) == 6 for i in range(len(b)))


def test_a_batch_that_ran_out_of_memory_runs_later_and_leaks_nothing(gastar):
    count = 64
    for warm in (True, False):  # the first time loads kernels
        before = _free()
        with gastar.Engine(0) as eng:
            b = _long_grids(eng, count)
            b.run()
            parts = _partitions(b, count)
            b.close()
            eng.server(budget_bytes=1 << 30).close()
            b = _long_grids(eng, count)
            hog = _fill(parts + 64 * MIB + 40 * MIB)  # the partitions fit, the paths do not
            with pytest.raises(gastar.GastarError, match="OUT_OF_MEMORY"):
                b.run()
            del hog
            _free()  # back from torch's cache
            c = _long_grids(eng, count + 8)
            c.run()
            assert _solved(c)
            c.close()
            b.run()
            assert _solved(b)
            b.close()
        after = _free()
    assert after >= before - 64 * MIB


def _puzzles(eng, gastar, count):
    """15-puzzles, whose partitions take about 100 MB each."""
    b = eng.batch()
    for i in range(count):
        b.add_sliding(*gastar.gen_sliding(4, 700 + i, 20, 24))
    return b


@pytest.fixture()
def kept(gastar):
    """An engine, and the bytes it holds after batches were closed."""
    with gastar.Engine(0) as eng:
        s, g = gastar.gen_sliding(4, 1, 20, 24)
        eng.solve_sliding(s, g, 4)
        before = _free()
        for _ in range(3):
            b = _puzzles(eng, gastar, 40)
            b.run()
            b.close()
        yield eng, before - _free()


def test_memory_kept_after_a_batch_serves_torch(kept):
    import torch
    eng, held = kept
    assert held > 2 << 30  # what this is about
    hog = _fill(512 * MIB)
    more = torch.empty(held - 512 * MIB, dtype=torch.uint8, device="cuda")  # more than is free
    del hog, more
    _free()


def test_memory_kept_after_a_batch_serves_the_library(kept, gastar):
    """Uploads, another context's solves and batches, and batches of the same
    context, when the rest of the device is taken."""
    import numpy as np
    eng, held = kept
    assert held > 2 << 30
    grid = np.full((20000, 50000), 3, dtype=np.uint8)  # 1 GB
    hog = _fill(512 * MIB)
    assert eng.grid_min_weight(grid)[0] == 3
    del hog
    _free()
    for _ in range(2):
        b = _puzzles(eng, gastar, 40)
        b.run()
        b.close()
    with gastar.Engine(0) as other:
        hog = _fill(512 * MIB)
        s, g = gastar.gen_sliding(4, 2, 20, 24)
        want = eng.solve_sliding(s, g, 4).cost
        r = other.solve_sliding(s, g, 4, table_log2=26)  # a 1 GiB table
        assert r.status_name == "OK" and r.cost == want
        b = _puzzles(other, gastar, 10)
        b.run()
        assert all(b.result(i).status_name == "OK" for i in range(len(b)))
        b.close()
        del hog
        _free()


def test_a_small_batch_leaves_the_rest_of_what_is_kept(kept, gastar):
    import torch
    eng, held = kept
    b = _puzzles(eng, gastar, 2)
    b.run()
    took = b.stats()["device_bytes"]
    assert took < 512 * MIB
    hog = _fill(512 * MIB)
    more = torch.empty(held - took - 512 * MIB, dtype=torch.uint8, device="cuda")
    assert b.result(0).status_name == "OK"
    b.rerun()
    assert b.result(0).status_name == "OK"
    del hog, more
    _free()
    b.close()


def test_batches_use_what_is_kept_when_the_device_is_full(kept, gastar):
    eng, held = kept
    hog = _fill(600 * MIB)
    for count in (40, 7, 40):
        b = _puzzles(eng, gastar, count)
        b.run()
        assert all(b.result(i).status_name == "OK" for i in range(count))
        b.close()
    del hog
    _free()


def test_a_servers_budget_counts_what_another_context_keeps(kept, gastar):
    eng, held = kept
    with gastar.Engine(0) as other:
        free = _free()
        budget = free + held - (3 << 30)
        srv = other.server(budget_bytes=budget, weights_pool=0)
        assert _free() <= free + held - budget
        i = srv.submit_sliding(*gastar.gen_sliding(3, 9, 20, 24))
        assert srv.drain([i])[i].status_name == "OK"
        srv.close()


def test_a_regrown_table_far_larger_than_needed_is_not_kept(gastar, oracle):
    """2^24 slots with a limit of a tenth of them, then eight times as many
    (2 GiB) where twice would have done."""
    kw = dict(table_log2=24, load_factor=0.1)
    with gastar.Engine(0) as eng:
        for walk in range(16, 30):  # boards whose blind search claims 1.8 to 3.2 M states
            s, g = gastar.gen_sliding(4, 800 + walk, walk, walk)
            claims = eng.solve_sliding(s, g, 4, heuristic=gastar.H_ZERO, table_log2=26).table_used
            if 1_800_000 < claims < 3_200_000:
                break
        assert 1_800_000 < claims < 3_200_000
    want = oracle.sliding_astar(4, s, g, path=False)[0].cost
    easy = gastar.gen_sliding(4, 1, 20, 24)
    with gastar.Engine(0) as eng:
        cost = eng.solve_sliding(*easy, 4, **kw).cost
        before = _free()
        for _ in range(2):
            r = eng.solve_sliding(s, g, 4, heuristic=gastar.H_ZERO, **kw)
            assert r.status_name == "OK" and r.cost == want and r.attempts == 2
            assert _free() > before - 1024 * MIB  # 2 GiB and its claim list before
            assert eng.solve_sliding(*easy, 4, **kw).cost == cost
    with gastar.Engine(0) as eng:  # a table that the caller asked for stays
        eng.solve_sliding(*easy, 4, table_log2=27)
        before = _free()
        r = eng.solve_sliding(s, g, 4, heuristic=gastar.H_ZERO, **kw)
        assert r.cost == want and r.attempts == 2
        assert abs(_free() - before) < 256 * MIB


def test_a_resident_batch_does_not_shrink_what_is_kept(gastar):
    """8.6 GB in a resident batch and 11.5 GB kept for the next: over the 16 GiB
    that are kept unused only together."""
    with gastar.Engine(0) as eng:
        for _ in range(2):
            b = _puzzles(eng, gastar, 80)
            b.run()
            b.close()
        resident = _puzzles(eng, gastar, 60)
        resident.run()
        b = _puzzles(eng, gastar, 80)
        b.run()
        held = _free()
        b.close()
        assert _free() < held + 512 * MIB
        resident.close()

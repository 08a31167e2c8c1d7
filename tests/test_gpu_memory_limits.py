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

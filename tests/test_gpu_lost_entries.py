"""Iterations that lose entries prove nothing, whatever else ended the search in
the same iteration: the status is the loss, not a budget's, and never OK."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = np.array([1, 2, 3, 4, 0, 5, 6, 7, 8], dtype=np.uint8)  # blank in the middle: four successors


def _moved(cell):
    b = START.copy()
    b[4], b[cell] = b[cell], 0
    return b


# One block (32 pops an iteration), a cluster (the default), a ring of 17 blocks.
SHAPES = {"block": dict(num_queues=32), "cluster": dict(),
          "ring": dict(num_queues=17 * 32, expansion_width=4, warps_per_block=8)}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("cell", [1, 3, 5, 7])
def test_a_full_table_is_not_masked_by_a_budget(engine, shape, cell):
    """Four slots hold the start and three of its four successors, in the
    iteration that is the budget's last."""
    kw = dict(table_log2=2, regrow=0, **SHAPES[shape])
    assert engine.solve_sliding(START, _moved(cell), 3, **kw).status_name == "TABLE_FULL"
    for budget in (dict(max_iterations=1), dict(max_expansions=1, max_iterations=1)):
        r = engine.solve_sliding(START, _moved(cell), 3, **budget, **kw)
        assert r.status_name == "TABLE_FULL"


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_budgets_alone_keep_their_status(engine, gastar, shape):
    s, g = gastar.gen_sliding(3, 5, 60, 60)
    assert engine.solve_sliding(s, g, 3, max_iterations=2, **SHAPES[shape]).status_name == "BUDGET"
    assert engine.solve_sliding(s, g, 3, max_expansions=3, **SHAPES[shape]).status_name == "BUDGET"

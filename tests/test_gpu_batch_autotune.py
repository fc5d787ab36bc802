"""The batch autotuner times what it returns: every candidate runs enough
iterations to launch its graph (the first and the last iteration of a run are
outside it), shapes that launch the same kernels are timed once, and the state
and the results do not depend on it."""
import pytest

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import BatchSolver
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu


def spots_of(count, hands):
    board = "Ks7s2dTh4c"
    return [abi.make_config(board, ranges(abi.parse_cards(board), hands, i, False), pot=700, stack=4000 + 300 * (i % 5),
                            menu_=abi.menu(["50%", "allin"], ["2.5x"]), storage=abi.STORAGE_F32, **workloads.DCFR)
            for i in range(count)]


# Short hand lists and many terminals: groups of warps; few terminals, or long hand lists: a block each.
@pytest.mark.parametrize("count,hands,groups", [(160, (90, 70), True), (4, (90, 70), False), (160, (1081, 900), False)])
@pytest.mark.parametrize("trial", [1, 4, 10])
def test_candidates_launch_their_graphs(gpu, count, hands, groups, trial):
    b = BatchSolver.new(spots_of(count, hands))
    b.iterate(3)
    before = b.kernel_launches()
    t = b.autotune(trial)
    launched = b.kernel_launches() - before
    # Two launches before an iteration, four in each.
    assert launched >= t.candidates * (2 + 4 * (trial + 2)), (launched, t.candidates)
    assert t.candidates > 4 if groups else t.candidates <= 4
    assert b.iterations() == 3 and 0 < t.trial_ms < 1e3
    b.iterate(30)
    c = BatchSolver.new(spots_of(count, hands))
    c.iterate(33)
    for i in (0, count - 1):
        assert all(bits_equal(x, y) for x, y in zip(b.download_storage(i), c.download_storage(i))), f"spot {i}"
    b.close()
    c.close()

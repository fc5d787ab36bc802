"""Which root streets take segment passes (segment.cu): few nodes a level. Wider
ones run level by level, where an iteration grows slowly with the tree; segment
passes took as many times longer as there are more nodes. Both sides of the rule
equal the oracle bit for bit in exact precision."""
import numpy as np
import pytest

from oracle_api import OracleSolver
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu

SMALL = (["33%", "66%", "100%", "allin"], ["2x", "4x", "allin"], 9000)  # 62 decisions on 5 levels
WIDE = (["20%", "40%", "60%", "80%", "100%", "130%", "160%", "allin"], ["2x", "4x", "allin"], 15000)  # 142


def river(menu, counts, precision):
    bets, raises, stack = menu
    board = "Ks7s2dTh4c"
    return abi.make_config(board, ranges(abi.parse_cards(board), counts, 5, False), pot=700, stack=stack,
                           menu_=abi.menu(bets, raises), storage=abi.STORAGE_F32, precision=precision, **workloads.DCFR)


def us(cfg):
    g = Solver.new(cfg)
    g.iterate(60)
    best = 1e9
    for _ in range(4):
        g.iterate(200)
        best = min(best, g.last_iterate_ms() * 5.0)
    g.close()
    return best


@pytest.mark.parametrize("hands", [200, 500])
def test_iteration_grows_slower_than_the_tree(gpu, hands):
    """2.3 times the decisions: 1.3 to 1.5 times as long by levels, 2.3 to 2.4 by segment passes."""
    assert us(river(WIDE, (hands, hands), "fast")) < 1.9 * us(river(SMALL, (hands, hands), "fast"))


@pytest.mark.parametrize("menu", [SMALL, WIDE])
@pytest.mark.parametrize("counts", [(33, 70), (200, 161)])
def test_both_sides_equal_the_oracle(gpu, menu, counts):
    cfg = river(menu, counts, "exact")
    o, g = OracleSolver(cfg), Solver.new(cfg)
    o.iterate(45)
    g.iterate(45)  # past the iterations that always run one by one
    assert all(bits_equal(x, y) for x, y in zip(g.download_storage(), o.storage()))
    assert g.exploitability() == o.exploitability()
    g.close()

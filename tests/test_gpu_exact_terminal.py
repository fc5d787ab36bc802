"""The exact terminal kernel (terminal.cu): bit for bit with the oracle at hand
counts around its unrolled chains (8 additions a step), on boards where every
hand ties or few do, with and without rake (tie payoffs), from a river and a
turn root (all-in runouts take the scalar evaluator)."""
import numpy as np
import pytest

from oracle_api import OracleSolver
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("board", ["AsKsQsJsTs", "2c2d2h2s3c", "9c8d7h6s2c", "Ks7s2dTh4c", "9c8d7h6s", "AhAd7c7s"])
@pytest.mark.parametrize("counts", [(2, 7), (8, 9), (16, 17), (63, 250), (700, 65)])
def test_exact_terminals_equal_the_oracle(gpu, board, counts):
    if len(board) == 8 and max(counts) > 300:
        counts = (150, 65)
    for rake in (0.0, 0.07):
        cfg = abi.make_config(board, ranges(abi.parse_cards(board), counts, 11, False), pot=900, stack=1500,
                              menu_=abi.menu(["60%", "allin"], ["allin"]), storage=abi.STORAGE_F32, precision="exact",
                              rake_rate=rake, rake_cap=150.0 if rake else 0.0, **workloads.DCFR)
        o = OracleSolver(cfg)
        o.iterate(4)
        g = Solver.new(cfg)
        g.iterate(4)
        assert all(bits_equal(a, b) for a, b in zip(g.download_storage(), o.storage()))
        assert g.exploitability() == o.exploitability()
        g.close()

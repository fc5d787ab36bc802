"""A solve looks at its cancel flag before every iteration (dcfr.h), whatever
it launches at once: cancelled from another thread at arbitrary moments, it
stops after any number of iterations, not only after whole graphs of them."""
import ctypes as C
import threading

import pytest

from poker_trainer_b200 import workloads
from poker_trainer_b200.solver import Solver, SolveOptions

pytestmark = pytest.mark.gpu


def test_cancelled_after_any_iteration(gpu):
    g = Solver.new(workloads.river_spot())
    g.iterate(100)  # past the iterations that always run one by one
    residues = set()
    for k in range(24):
        g.set_iterations(0)
        flag = C.c_int32(0)
        timer = threading.Timer(0.004 + 0.0013 * k, lambda: setattr(flag, "value", 1))
        timer.start()
        g.solve(SolveOptions(max_iterations=200_000, target_exploitability_pct=0.0, check_every=200_000),
                cancel=flag)
        timer.join()
        residues.add(g.iterations() % 10)
    g.close()
    # 24 solves that stop anywhere all share a residue with probability 1e-23.
    assert len(residues) > 1, residues

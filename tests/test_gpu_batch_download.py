"""Reading spots' storage from a batch: by several threads at once, for a spot
whose storage takes several rounds of the transfer block, and on a fresh batch
at the cost of any later read."""
import time
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import BatchSolver, Solver
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workers", [2, 8])
def test_threads_read_their_own_spots(gpu, workers):
    cfgs = workloads.batched_river_spots(count=24, seed=5)
    b = BatchSolver.new(cfgs)
    b.iterate(3)
    spots = list(range(24)) * 8
    with ThreadPoolExecutor(workers) as pool:
        got = list(pool.map(b.download_storage, spots))
    want = [b.download_storage(i) for i in range(24)]
    for i, (r, s) in zip(spots, got):
        assert np.array_equal(r, want[i][0]) and np.array_equal(s, want[i][1]), f"spot {i}"
    b.close()


@pytest.mark.parametrize("counts", [(1, 1), (61, 47), (1081, 300)])
def test_large_spot(gpu, counts):
    """2552 decision nodes: 0.1 to 40 MB of storage."""
    cfg = abi.make_config("Ks7s2dTh4c", ranges(abi.parse_cards("Ks7s2dTh4c"), counts, 3, False), pot=400, stack=16084,
                          menu_=abi.menu(["55%", "100%", "115%", "150%", "allin"],
                                         ["2.1x", "2.2x", "4.0x", "4.1x", "4.8x", "allin"], max_raises=7),
                          storage=abi.STORAGE_F32, **workloads.DCFR)
    b, g = BatchSolver.new([cfg]), Solver.new(cfg)
    b.iterate(4)
    g.iterate(4)
    assert all(bits_equal(x, y) for x, y in zip(b.download_storage(0), g.download_storage()))
    b.close()
    g.close()


def test_first_read_costs_what_a_later_one_does(gpu):
    cfgs = workloads.batched_river_spots(count=64, seed=9)
    first, later = [], []
    for _ in range(6):
        b = BatchSolver.new(cfgs)
        b.iterate(2)
        for times in (first, later):
            t = time.perf_counter()
            b.download_storage(0)
            times.append(time.perf_counter() - t)
        b.close()
    # The least of six handles: what is made once a process, and the host's noise, are not in it. A table and
    # buffers per batch took 20 times a later read.
    assert min(first) < 4 * min(later), (first, later)

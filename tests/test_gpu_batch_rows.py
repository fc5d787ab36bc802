"""The batch's row passes (batch.cu) and its terminals over spots of different
hand counts: every spot bit for bit with a single solve of it, at hand counts
around a slice's edge, with slices that reach nothing, at each instantiation's
action counts, and with so many spots that every warp takes its own slice."""
import numpy as np
import pytest

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import BatchSolver, Solver
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu

BOARDS = ["Ks7s2dTh4c", "AhAd8c3s3h", "5h6h7hTcJd"]
MENUS = {4: (["50%", "allin"], ["2.5x"]), 8: (["33%", "66%", "100%", "allin"], ["2x", "4x", "allin"]),
         16: (["20%", "40%", "60%", "80%", "100%", "130%", "160%", "allin"], ["2x"])}


def spot(i, counts, maxa, holes, rake):
    board = BOARDS[i % len(BOARDS)]
    return abi.make_config(board, ranges(abi.parse_cards(board), counts, 100 + i, holes), pot=500 + 100 * (i % 7),
                           stack=3000 + 500 * (i % 5), menu_=abi.menu(*MENUS[maxa]), storage=abi.STORAGE_F32,
                           rake_rate=rake, rake_cap=200.0 if rake else 0.0, **workloads.DCFR)


def check(cfgs, iterations, some):
    b = BatchSolver.new(cfgs)
    b.iterate(iterations)
    e = b.exploitability()
    for i in some:
        g = Solver.new(cfgs[i])
        g.iterate(iterations)
        assert all(bits_equal(x, y) for x, y in zip(b.download_storage(i), g.download_storage())), f"spot {i}"
        assert e[i] == g.exploitability(), f"spot {i}"
        g.close()
    b.close()


@pytest.mark.parametrize("maxa", list(MENUS))
@pytest.mark.parametrize("rake", [0.0, 0.05])
def test_uneven_spots_equal_single_solves(gpu, maxa, rake):
    counts = [(3, 5), (31, 33), (32, 64), (95, 129), (300, 161), (65, 700)]
    cfgs = [spot(i, c, maxa, i % 2 == 1, rake) for i, c in enumerate(counts)]
    check(cfgs, 13, range(len(cfgs)))


def test_a_slice_per_warp(gpu):
    """112 spots of 34 slices: past the rule's line for sharing a slice."""
    cfgs = [spot(i, (1081 - i, 900 + i) if i else (1081, 1081), 4, i % 3 == 0, 0.0) for i in range(112)]
    check(cfgs, 6, (0, 1, 57, 111))


def test_many_short_spots(gpu):
    """Short hand lists and many spots: the two-warps-per-terminal kernel over units of different spots."""
    cfgs = [spot(i, (20 + i % 90, 130 - i % 90), 8, False, 0.0) for i in range(160)]
    check(cfgs, 9, (0, 80, 159))

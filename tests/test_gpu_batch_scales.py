"""Batched spots whose two ranges differ in length and in scale: a terminal's
fixed-point scale is set by its own opponent's row, so every spot is bit for
bit a single solve of it, and reading the exploitability between iterations
changes nothing."""
import pytest

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import BatchSolver, Solver
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu

BOARDS = ["Ks7s2dTh4c", "AhAd8c3s3h", "5h6h7hTcJd"]
# Hand counts of the players, and which of them holds the small weights.
COUNTS = [(65, 700, 0), (700, 65, 1), (161, 300, 0), (300, 161, 1), (8, 1000, 0), (200, 200, 0)]


def spot(i, small):
    n0, n1, who = COUNTS[i % len(COUNTS)]
    board = BOARDS[i % len(BOARDS)]
    r = ranges(abi.parse_cards(board), (n0, n1), 40 + i, False)
    r[who] = (r[who] * small).astype("float32")
    return abi.make_config(board, r, pot=500 + 100 * (i % 7), stack=3000 + 500 * (i % 5),
                           menu_=abi.menu(["50%", "allin"], ["2.5x"]), storage=abi.STORAGE_F32, **workloads.DCFR)


# Six spots: a block per terminal. 240 short ones: groups of warps.
@pytest.mark.parametrize("count", [6, 240])
@pytest.mark.parametrize("small", [1e-6, 1e-9, 1e-12])
def test_ranges_of_different_scales(gpu, count, small):
    cfgs = [spot(i, small) for i in range(count)]
    b, c = BatchSolver.new(cfgs), BatchSolver.new(cfgs)
    b.iterate(11)
    for n in (3, 1, 7):
        c.iterate(n)
        e = c.exploitability()
    for i in range(0, count, max(1, count // 6 + 1)):
        g = Solver.new(cfgs[i])
        g.iterate(11)
        single = g.download_storage()
        assert all(bits_equal(x, y) for x, y in zip(b.download_storage(i), single)), f"spot {i}"
        assert all(bits_equal(x, y) for x, y in zip(c.download_storage(i), single)), f"spot {i}, checks between"
        assert e[i] == g.exploitability(), f"spot {i}"
        g.close()
    b.close()
    c.close()

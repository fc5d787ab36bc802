"""Batched spots at the slot limit (4096 reach slots a traversal): trees whose
plan records do not fit shared memory are solved, bit for bit as single solves,
and larger ones are refused."""
import pytest

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import BatchSolver, Solver, SolverError
from test_gpu_segment import bits_equal, ranges

pytestmark = pytest.mark.gpu

# bets, raises, most raises, pot, stack: 8,049 to 8,181 nodes; the last ones need more slots.
LARGE = [(["10%", "25%", "40%", "90%", "100%", "allin"], ["3.4x", "3.6x", "3.8x", "allin"], 7, 400, 70324),
         (["15%", "30%", "125%", "130%", "145%", "allin"], ["4.0x", "4.4x", "4.8x", "5.2x", "allin"], 6, 700, 85926),
         (["35%", "45%", "65%", "120%", "150%", "allin"], ["2.3x", "3.9x", "4.9x", "5.5x", "allin"], 7, 1000, 83027)]
TOO_LARGE = (["75%", "100%", "120%", "125%", "145%", "155%", "allin"], ["2.4x", "3.0x", "3.2x", "3.8x", "allin"], 5,
             700, 54344)
SMALL = (["50%", "allin"], ["2.5x"], 3, 700, 4000)


def spot(tree, counts, seed=1):
    bets, raises, most, pot, stack = tree
    board = "Ks7s2dTh4c"
    return abi.make_config(board, ranges(abi.parse_cards(board), counts, seed, False), pot=pot, stack=stack,
                           menu_=abi.menu(bets, raises, max_raises=most), storage=abi.STORAGE_F32, **workloads.DCFR)


def check(cfgs, some):
    b = BatchSolver.new(cfgs)
    b.iterate(5)
    e = b.exploitability()
    for i in some:
        g = Solver.new(cfgs[i])
        g.iterate(5)
        assert all(bits_equal(x, y) for x, y in zip(b.download_storage(i), g.download_storage())), f"spot {i}"
        assert e[i] == g.exploitability(), f"spot {i}"
        g.close()
    b.close()


@pytest.mark.parametrize("tree", LARGE)
@pytest.mark.parametrize("counts", [(31, 50), (300, 97)])
def test_largest_trees(gpu, tree, counts):
    check([spot(tree, counts)], [0])


def test_a_large_tree_among_small_ones(gpu):
    """So many slices that a warp takes each alone."""
    cfgs = [spot(SMALL, (1081, 1000), i) for i in range(111)] + [spot(LARGE[0], (97, 200))]
    check(cfgs, [0, 60, 111])


def test_past_the_slot_limit(gpu):
    with pytest.raises(SolverError) as e:
        BatchSolver.new([spot(TOO_LARGE, (31, 50))])
    assert e.value.code == abi.ERR_UNSUPPORTED


def device_bytes(cfgs):
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    b = BatchSolver.new(cfgs)
    taken = before - torch.cuda.mem_get_info()[0]
    b.close()
    return taken


def test_narrow_spots_beside_a_wide_one(gpu):
    """A spot's rows are as long as its own ranges. What is common to a batch is
    about 105 KB a spot of 1081 hands (its scan layouts), and the arrays are
    allocated in pieces of 2 MB."""
    tree = (["50%", "100%", "allin"], ["50%", "100%", "allin"], 3, 700, 9000)
    narrow = [spot(tree, (60, 47), i) for i in range(480)]
    wide = [spot(SMALL, (1081, 1000))]
    device_bytes(wide)  # the context's own
    apart = device_bytes(narrow) + device_bytes(wide)
    assert device_bytes(narrow + wide) <= apart + (len(narrow) + 1) * 110_000 + (24 << 20)

"""Which trees the tile terminal kernel runs: by request where the hand lists
allow tiles (16 terminals up to 512 hands, 8 up to about 1000), and by default
from 384 terminals an SM; the width is reported, so that a comparison with
another kernel (test_gpu_tile_terminal.py) is known to be one."""
import numpy as np
import pytest

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver
from test_gpu_segment import ranges
from test_gpu_terminal_kernels import same_bits
from test_gpu_tile_terminal import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(CASES))
def test_width_by_hand_lists(gpu, name, monkeypatch):
    monkeypatch.setenv("DCFR_TERMINAL_KERNEL", "tile")
    g = Solver.new(CASES[name]())
    most = max(len(g.hands(p)[0]) for p in (0, 1))
    assert most <= 1000 or most > 1024
    want = ("group", 16) if most <= 512 else ("group", 8) if most <= 1000 else ("block", 0)
    assert g.terminal_kernel() == want
    g.close()


def flop(cards, counts):
    """A flop with sampled deals: 62,000 terminals and more at five cards a street, 419 an SM."""
    board = "Ks7s2d"
    return abi.make_config(board, ranges(abi.parse_cards(board), counts, 4, False), pot=600, stack=9700,
                           menu_=abi.menu(["50%", "100%", "allin"], ["2.5x"]), storage=abi.STORAGE_F32,
                           sampled=(cards, cards, 3), **workloads.DCFR)


def outputs(cfg):
    g = Solver.new(cfg)
    g.iterate(3)
    out = (*g.download_storage(), np.array([g.exploitability()]))
    kernel = g.terminal_kernel()
    g.close()
    return kernel, out


@pytest.mark.parametrize("counts,width", [((300, 250), 16), ((700, 90), 8)])
def test_default_by_terminals(gpu, counts, width, monkeypatch):
    monkeypatch.delenv("DCFR_TERMINAL_KERNEL", raising=False)
    kernel, got = outputs(flop(5, counts))
    assert kernel == ("group", width)
    assert outputs(flop(3, counts))[0] == ("group", 0)
    monkeypatch.setenv("DCFR_TERMINAL_KERNEL", "warp")
    kernel, ref = outputs(flop(5, counts))
    assert kernel == ("warp", 0)
    assert all(same_bits(a, b) for a, b in zip(got, ref))

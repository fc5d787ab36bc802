"""The tile terminal kernel (terminal_tile.cu), bit for bit with the
warp-per-terminal kernel: at hand counts around its tile widths, runs and
loads (16 terminals a tile up to about 500 hands, 8 up to about 1000, none
above), in every traversal mode, with and without rake, chops and all-in
runouts, from storage with dead subtrees in it, and on tiles that no block
fills."""
import numpy as np
import pytest

import spots
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver
from test_gpu_segment import ranges
from test_gpu_terminal_kernels import random_storage, same_bits

pytestmark = pytest.mark.gpu


def turn(counts, rake=0.0, board="Ks7s2dTh", stack=3000, bets=("50%", "allin"), holes=False):
    return abi.make_config(board, ranges(abi.parse_cards(board), counts, 5, holes), pot=900, stack=stack,
                           menu_=abi.menu(list(bets), ["2.5x"]), storage=abi.STORAGE_F32, rake_rate=rake,
                           rake_cap=150.0 if rake else 0.0, **workloads.DCFR)


CASES = {
    "few": lambda: turn((5, 9)),
    "edges 63 65": lambda: turn((63, 65), rake=0.06),
    "edges 127 129": lambda: turn((127, 129)),
    "uneven": lambda: turn((40, 500), rake=0.06, holes=True),
    "wide 16": lambda: turn((512, 400)),
    "wide 8": lambda: turn((521, 700), rake=0.06),
    "runs 8": lambda: turn((1000, 960)),
    "ties": lambda: turn((200, 180), board="AcAdAhAs", rake=0.06),
    "narrow turn": workloads.turn_narrow_spot,
    "turn": workloads.turn_spot,
    "river": workloads.river_spot,
    "iso turn": spots.iso_turn_config,
    "all-in turn": spots.allin_turn_config,
    "mid street raked": lambda: spots.mid_street_config(True),
}


def outputs(make, kernel, monkeypatch):
    monkeypatch.setenv("DCFR_TERMINAL_KERNEL", kernel)
    g = Solver.new(make())
    out = {}
    r, s = random_storage(g.storage_len(), 11)
    for p in (0, 1):
        for mode in (abi.MODE_BEST_RESPONSE, abi.MODE_AVERAGE, abi.MODE_CFR):
            g.upload_storage(r, s)
            out[f"traverse p={p} mode={mode}"] = np.asarray(g.traverse(p, mode, 3), np.float32).copy()
            out[f"storage p={p} mode={mode}"] = np.concatenate(g.download_storage())
    g.close()
    g = Solver.new(make())
    g.iterate(25)  # pure strategies by then: dead subtrees
    out["storage"] = np.concatenate(g.download_storage())
    out["exploitability"] = np.array([g.exploitability()])
    out["root"] = np.asarray(g.query(()).ev)
    g.close()
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_tiles_equal_the_warp_kernel(gpu, name, monkeypatch):
    ref = outputs(CASES[name], "warp", monkeypatch)
    got = outputs(CASES[name], "tile", monkeypatch)
    for key in ref:
        assert same_bits(got[key], ref[key]), f"{name}: {key}"

"""Fused segments (fused.cu): one block walks the decision nodes of a street's
subtree, its tasks, liveness and storage in shared memory. Exact precision
must equal the oracle bit for bit, with f32 and with 16-bit storage, at hand
counts around a thread's 4 hands and a warp's 128, at each instantiation's
action counts, where parts of the segments are dead, from the smallest
segments to the largest that run fused, and past them."""
import numpy as np
import pytest

from oracle_api import OracleSolver
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver

pytestmark = pytest.mark.gpu


def ranges(board, counts, seed, holes):
    rng = np.random.default_rng(seed)
    free = [i for i in range(1326) if not set(abi.combo_cards(i)) & set(board)]
    out = []
    for n in counts:
        r = np.zeros(1326, np.float32)
        ids = [free[i] for i in sorted(rng.choice(len(free), n, replace=False).tolist())]
        r[ids] = 0.05 + 0.95 * rng.random(n).astype(np.float32)
        if holes:  # nearly all of the range vanishes after a few splits
            r[ids[3:]] = 1e-42
        out.append(r)
    return out


CASES = [
    # hands, root bets and raises, later bets and raises, stack, holes
    ((1, 2), ["allin"], [], ["allin"], [], 900, False),
    ((127, 129), ["50%"], ["allin"], ["50%", "allin"], ["allin"], 3000, False),
    ((128, 4), ["50%"], ["allin"], ["33%", "75%", "allin"], ["2.5x"], 4000, True),
    # Up to 8 and up to 16 actions.
    ((60, 130), ["50%"], ["allin"], ["20%", "40%", "60%", "80%", "allin"], ["allin"], 2500, True),
    ((33, 41), ["50%"], ["allin"], ["15%", "25%", "35%", "45%", "55%", "65%", "75%", "allin"], [], 4000,
     False),
    # Segments of tens of nodes, and some past 48 (level by level).
    ((20, 90), ["50%"], [], ["25%", "50%", "75%", "allin"], ["2.5x", "allin"], 2500, False),
    ((20, 90), ["50%"], [], ["25%", "50%", "75%", "100%", "allin"], ["2.2x", "3x", "allin"], 9000, True),
    ((1128, 1127), ["allin"], [], ["60%"], ["allin"], 1500, False),
]


@pytest.mark.parametrize("storage", ["f32", "compressed"])
@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("unweighted", [True, False])
def test_fused_segments_equal_the_oracle(gpu, case, storage, unweighted):
    counts, bets, raises, later, reraises, stack, holes = CASES[case]
    board = "Ks7s2dTh"
    cfg = abi.make_config(board, ranges(abi.parse_cards(board), counts, 11 + case, holes), pot=600, stack=stack,
                          menu_=abi.menu(bets, raises), future_menu=abi.menu(later, reraises),
                          storage=abi.STORAGE_F32 if storage == "f32" else abi.STORAGE_COMPRESSED, precision="exact",
                          **dict(workloads.DCFR, unweighted_average=unweighted))
    o, g = OracleSolver(cfg), Solver.new(cfg)
    for its in (1, 4):
        o.iterate(its)
        g.iterate(its)
        if storage == "f32":
            a, b = g.download_storage(), o.storage()
        else:
            a, b = g.download_storage_compressed(), o.compressed_storage()
        for x, y in zip(a, b):
            x, y = np.asarray(x), np.asarray(y)
            same = (x == y) if x.dtype != np.float32 else (x.view(np.uint32) == y.view(np.uint32)) | ((x == 0) & (y == 0))
            assert x.shape == y.shape and bool(np.all(same))
    assert g.exploitability() == o.exploitability()
    g.close()

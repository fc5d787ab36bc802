"""Segment passes (segment.cu): the root street's decision nodes by slices of
32 hands, with the strategy sums of nodes that a slice does not reach put off
to the up pass. Exact precision must equal the oracle bit for bit (the
kernels' operations are the reference's in its order) at hand counts around a
slice's edge, with slices that reach nothing, at each instantiation's action
counts, on the root street of a turn game, and where the segment is too large
for the passes and runs level by level."""
import numpy as np
import pytest

from oracle_api import OracleSolver
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver

pytestmark = pytest.mark.gpu


def bits_equal(a, b):
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return a.shape == b.shape and bool(np.all((a.view(np.uint32) == b.view(np.uint32)) | ((a == 0) & (b == 0))))


def ranges(board, counts, seed, holes):
    """Ranges of counts[p] hands off the board; `holes` puts a run of 40 hands
    at a weight that vanishes beside the others after a few splits."""
    rng = np.random.default_rng(seed)
    free = [i for i in range(1326) if not set(abi.combo_cards(i)) & set(board)]
    out = []
    for n in counts:
        r = np.zeros(1326, np.float32)
        ids = sorted(rng.choice(len(free), n, replace=False).tolist())
        r[[free[i] for i in ids]] = 0.05 + 0.95 * rng.random(n).astype(np.float32)
        if holes and n > 80:
            r[[free[i] for i in ids[20:60]]] = 1e-42
        out.append(r)
    return out


CASES = [
    # hands, bets, raises, stack, board, holes
    ((1, 1), ["allin"], ["allin"], 1000, "Ks7s2dTh4c", False),
    ((31, 33), ["50%", "allin"], ["2.5x"], 4000, "Ks7s2dTh4c", False),
    ((32, 64), ["50%", "100%", "allin"], ["2.5x"], 9000, "Ks7s2dTh4c", False),
    ((95, 129), ["33%", "66%", "100%", "allin"], ["2x", "4x", "allin"], 9000, "AhAd8c3s3h", True),
    ((400, 161), ["20%", "40%", "60%", "80%", "100%", "130%", "160%", "allin"], ["2x"], 7000, "5h6h7hTcJd", True),
    ((1081, 1081), ["50%", "100%", "allin"], ["2.5x"], 9000, "Ks7s2dTh4c", False),
    ((97, 50), ["33%", "allin"], ["2.5x"], 3000, "Ks7s2dTh", True),
    # Hundreds of decision nodes: past the passes' shared memory.
    ((40, 70), ["15%", "30%", "45%", "60%", "75%", "allin"], ["2.1x", "2.6x", "3.2x", "4x", "allin"], 15000,
     "Ks7s2dTh4c", False),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("rake", [0.0, 0.05])
def test_segment_passes_equal_the_oracle(gpu, case, rake):
    counts, bets, raises, stack, board, holes = CASES[case]
    cfg = abi.make_config(board, ranges(abi.parse_cards(board), counts, 7 + case, holes), pot=700, stack=stack,
                          menu_=abi.menu(bets, raises), storage=abi.STORAGE_F32, precision="exact", rake_rate=rake,
                          rake_cap=200.0 if rake else 0.0, **workloads.DCFR)
    its = 12
    o = OracleSolver(cfg)
    o.iterate(its)
    ro, so = o.storage()
    g = Solver.new(cfg)
    g.iterate(its)
    rg, sg = g.download_storage()
    assert bits_equal(rg, ro) and bits_equal(sg, so)
    assert g.exploitability() == o.exploitability()
    # Single traversals (the same passes, one direction a launch).
    assert g.iterations() == its
    g.iterate(3)
    o.iterate(3)
    rg, sg = g.download_storage()
    ro, so = o.storage()
    assert bits_equal(rg, ro) and bits_equal(sg, so)
    g.close()


def test_reach_weighted_average(gpu):
    """The average weighted by reach: deferred sums add nothing but decay."""
    cfg = abi.make_config("Ks7s2dTh4c", ranges(abi.parse_cards("Ks7s2dTh4c"), (200, 150), 3, True), pot=700, stack=5000,
                          menu_=abi.menu(["50%", "allin"], ["2.5x"]), storage=abi.STORAGE_F32, precision="exact",
                          **dict(workloads.DCFR, unweighted_average=False))
    o = OracleSolver(cfg)
    o.iterate(15)
    g = Solver.new(cfg)
    g.iterate(15)
    assert all(bits_equal(a, b) for a, b in zip(g.download_storage(), o.storage()))
    assert g.exploitability() == o.exploitability()
    g.close()

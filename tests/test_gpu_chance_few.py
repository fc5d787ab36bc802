"""Chance nodes of a layer that has few of them (kernels.cu,
chance_down_kernel and chance_up_kernel): splits by groups of children, sums
by a thread per hand with the isomorphic cards added after the dealt ones.
Exact precision must equal the oracle bit for bit (the sums' additions are the
reference's in its order) at hand counts around a block's and a thread's edge,
with no, some and many isomorphic cards, and where deals are sampled, so that
the last group of children is short."""
import numpy as np
import pytest

from oracle_api import OracleSolver
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import Solver

pytestmark = pytest.mark.gpu


def bits_equal(a, b):
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return a.shape == b.shape and bool(np.all((a.view(np.uint32) == b.view(np.uint32)) | ((a == 0) & (b == 0))))


def suit_closed(board, n, seed):
    """A range of at least n hands with every suit form of each, weighted alike
    (isomorphic cards need ranges that the suits' exchange leaves alone)."""
    rng = np.random.default_rng(seed)
    r = np.zeros(1326, np.float32)
    blocked = set(board)
    while np.count_nonzero(r) < n:
        cls = int(rng.integers(169))
        f = np.zeros(169, np.float32)
        f[cls] = 0.05 + 0.95 * rng.random()
        x = workloads.expand_classes(f).astype(np.float32)
        ids = [i for i in np.flatnonzero(x) if not set(abi.combo_cards(int(i))) & blocked]
        r[ids] = x[ids]
    return r


def some(board, n, seed):
    rng = np.random.default_rng(seed)
    free = [i for i in range(1326) if not set(abi.combo_cards(i)) & set(board)]
    r = np.zeros(1326, np.float32)
    ids = [free[i] for i in rng.choice(len(free), n, replace=False)]
    r[ids] = 0.05 + 0.95 * rng.random(n).astype(np.float32)
    return r


CASES = [
    ("Ks7s2dTh", (63, 65), some, {}),
    ("Ks7s2dTh", (1, 64), some, {}),
    ("Qd9d4c4h", (60, 129), suit_closed, {}),
    ("Ks7s2s2d", (250, 70), suit_closed, {}),
    ("KsQsJsTs", (64, 300), suit_closed, {}),
    ("Ks7s2d", (20, 33), some, dict(sampled=(3, 5, 7))),
    ("Ks7s2d", (12, 9), some, dict(sampled=(9, 2, 5))),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_chance_nodes_equal_the_oracle(gpu, case):
    board, counts, pick, deals = CASES[case]
    cards = abi.parse_cards(board)
    cfg = abi.make_config(board, [pick(cards, n, 31 * case + k) for k, n in enumerate(counts)], pot=600, stack=1500,
                          menu_=abi.menu(["60%"], ["allin"]), storage=abi.STORAGE_F32, precision="exact", **deals,
                          **workloads.DCFR)
    o, g = OracleSolver(cfg), Solver.new(cfg)
    o.iterate(4)
    g.iterate(4)
    ro, so = o.storage()
    rg, sg = g.download_storage()
    assert bits_equal(rg, ro) and bits_equal(sg, so)
    assert g.exploitability() == o.exploitability()
    g.close()

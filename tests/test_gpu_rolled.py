"""Iterations chained across their ends (Engine::enqueue_rolled): the up pass
that ends one and the down pass that begins the next share a launch, and the
terminal kernels clear the liveness flags and step the discounts. Chained
iterations must leave the storage of the same iterations launched one by one,
bit for bit, and in exact precision the oracle's: with each terminal kernel
that steps the discounts, across a restart of the average, after the iteration
is set, and where subtrees die and come back."""
import numpy as np
import pytest

from oracle_api import OracleSolver
from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.solver import BatchSolver, Solver

pytestmark = pytest.mark.gpu

SINGLES = 32  # iterations that a handle runs one by one before it chains them, ten at a time


def bits_equal(a, b):
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return a.shape == b.shape and bool(np.all((a.view(np.uint32) == b.view(np.uint32)) | ((a == 0) & (b == 0))))


def ranges(board, counts, seed):
    rng = np.random.default_rng(seed)
    free = [i for i in range(1326) if not set(abi.combo_cards(i)) & set(board)]
    out = []
    for n in counts:
        r = np.zeros(1326, np.float32)
        ids = [free[i] for i in rng.choice(len(free), n, replace=False)]
        r[ids] = 0.05 + 0.95 * rng.random(n).astype(np.float32)
        r[ids[: n // 3]] = 1e-42
        out.append(r)
    return out


def config(board, counts, precision, **dcfr):
    return abi.make_config(board, ranges(abi.parse_cards(board), counts, 5), pot=700, stack=5000,
                           menu_=abi.menu(["50%", "allin"], ["2.5x"]), storage=abi.STORAGE_F32, precision=precision,
                           **dict(workloads.DCFR, **dcfr))


@pytest.mark.parametrize("unweighted", [True, False])
@pytest.mark.parametrize("counts", [(90, 61), (400, 1081)])
def test_chained_iterations_equal_the_oracle(gpu, counts, unweighted):
    cfg = config("Ks7s2dTh4c", counts, "exact", unweighted_average=unweighted)
    o, g = OracleSolver(cfg), Solver.new(cfg)
    for its in (SINGLES, 30, 7, 40):
        o.iterate(its)
        g.iterate(its)
        assert all(bits_equal(a, b) for a, b in zip(g.download_storage(), o.storage()))
    assert g.exploitability() == o.exploitability()
    g.close()


@pytest.mark.parametrize("board, counts, kernel", [
    ("Ks7s2dTh4c", (300, 280), None),   # a block per terminal
    ("Ks7s2dTh", (61, 90), None),       # the default of a turn
    ("Ks7s2dTh", (61, 90), "group"),
    ("Ks7s2dTh", (61, 90), "exact"),
])
def test_chained_iterations_equal_single_ones(gpu, board, counts, kernel, monkeypatch):
    precision = "exact" if kernel == "exact" else "fast"
    if kernel == "group":
        monkeypatch.setenv("DCFR_TERMINAL_KERNEL", kernel)
    cfg = config(board, counts, precision)
    a, b = Solver.new(cfg), Solver.new(cfg)
    for its in (SINGLES, 20, 30):
        a.iterate(its)
        for _ in range(its):
            b.iterate(1)
        assert all(bits_equal(x, y) for x, y in zip(a.download_storage(), b.download_storage()))
    # Set back to an early iteration: discounts and the average's restart again.
    for s in (a, b):
        s.set_iterations(3)
    a.iterate(20)
    for _ in range(20):
        b.iterate(1)
    assert all(bits_equal(x, y) for x, y in zip(a.download_storage(), b.download_storage()))
    assert a.exploitability() == b.exploitability()
    a.close()
    b.close()


def test_chained_batch_iterations_equal_single_ones(gpu):
    cfgs = [config(board, counts, "fast") for board, counts in
            (("Ks7s2dTh4c", (90, 61)), ("AhAd8c3s3h", (300, 33)), ("5h6h7hTcJd", (1, 400)))]
    a, b = BatchSolver.new(cfgs), BatchSolver.new(cfgs)
    for its in (1, 2, 3, 27, 60):
        a.iterate(its)
        for _ in range(its):
            b.iterate(1)
        for k in range(len(cfgs)):
            assert all(bits_equal(x, y) for x, y in zip(a.download_storage(k), b.download_storage(k)))
    assert np.array_equal(a.exploitability(), b.exploitability())

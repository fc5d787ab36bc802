"""dcfr_showdown_values_noalloc called for many boards and hand lists in a row
on one stream: each call's values are those of the call alone, although all use
one static scratch, whose layout each call writes just before it is read."""
import ctypes as C

import numpy as np
import pytest

from poker_trainer_b200 import abi
from test_zz_no_alloc import cards_of, entry

pytestmark = pytest.mark.gpu


def test_calls_in_a_row(gpu):
    import torch

    f = entry()
    rng = np.random.default_rng(2)
    calls = []
    for k in range(60):
        board = rng.choice(52, 5, replace=False).astype(np.uint8)
        free = [i for i in range(abi.NUM_COMBOS) if not set(abi.combo_cards(i)) & set(board.tolist())]
        lists = [cards_of(sorted(rng.choice(free, n, replace=False).tolist()))
                 for n in (int(rng.integers(1, 1082)), (1, 40, 400, 1081)[k % 4])]
        reach = torch.tensor(rng.random(len(lists[1])).astype(np.float32), device="cuda")
        calls.append((np.ascontiguousarray(board), *lists, reach, float(rng.random()), -float(rng.random()), 0.25))

    def run(call):
        board, hero, opp, reach, win, lose, tie = call
        out = torch.full((len(hero),), float("nan"), dtype=torch.float32, device="cuda")
        rc = f(board.ctypes.data, hero.ctypes.data, len(hero), opp.ctypes.data, len(opp), reach.data_ptr(), win, lose,
               tie, out.data_ptr(), None)
        assert rc == abi.OK
        return out

    alone = []
    for call in calls:
        torch.cuda.synchronize()
        alone.append(run(call).cpu().numpy())
    torch.cuda.synchronize()
    for _ in range(5):
        outs = [run(call) for call in calls]
        torch.cuda.synchronize()
        for i, (got, want) in enumerate(zip(outs, alone)):
            assert np.all(np.isfinite(want)) and np.array_equal(got.cpu().numpy(), want), f"call {i}"

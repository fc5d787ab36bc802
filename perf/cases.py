"""What the performance of this framework is measured on: postflop solves of
every street and option, batched river solves, and the leaf network with the
depth-limited solve it serves, each through the public Python API.

A solve pass is what a study or review program does with a spot it holds
open: solve it for a number of iterations with exploitability checks on the
way, then read the root's strategies and EVs (and, where the program keeps
the solution, the whole storage). Every pass starts the DCFR schedule at its
first iteration, whose discounts clear the average and the positive regrets,
so passes on one handle do the same work.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from poker_trainer_b200 import abi, workloads
from poker_trainer_b200.leafdata import IN_DIM, OUT_DIM
from poker_trainer_b200.mlp import LeafNet
from poker_trainer_b200.solver import BatchSolver, Solver, SolveOptions

SOLVE = dict(kind="solve", ranges="uniform", keep=169, pot=2000, stack=9000, bets="50%,100%,allin", raises="2.5x",
             storage="f32", precision="fast", deal_turn=0, deal_river=0, rake=0.0, iterations=10, check_every=10,
             keep_storage=False)


def solve(**over):
    return dict(SOLVE, **over)


def listed():
    small = dict(bets="33%,75%,allin", raises="2.5x")
    flop = dict(ranges="dirichlet", keep=68, bets="33%,75%,allin", raises="3x")
    return [
        # The smallest call: a live review of a river decision between tight ranges.
        solve(name="river_quick", board="Ah8d3s3cJc", ranges="dirichlet", keep=40, pot=1350, stack=2475,
              bets="75%,allin", raises="3x"),
        # The river subgame of the benchmark with every hand, solved properly and kept.
        solve(name="river_wide", board="Ks7s2dTh4c", iterations=100, check_every=25, keep_storage=True),
        # The same subgame in the precision that reproduces the CPU solver bit for bit.
        solve(name="river_exact", board="Ks7s2dTh4c", precision="exact"),
        # The turn subgame of the benchmark: wide ranges, 48 rivers; the solution is kept.
        solve(name="turn_wide", board="Ks7s2dTh", keep=118, iterations=40, check_every=20, keep_storage=True, **small),
        # A raked turn spot with narrow ranges: chops, rake and average-strategy traversals in each check.
        solve(name="turn_raked", board="Qd9d4c4h", ranges="dirichlet", keep=68, pot=1830, stack=7400, rake=0.05,
              iterations=40, check_every=10, **small),
        # A flop explored quickly: sampled turn and river cards.
        solve(name="flop_sampled", board="Ks7s2d", pot=600, stack=9700, deal_turn=8, deal_river=6, iterations=20, **flop),
        # A three-bet pot on the flop with every card dealt; the default storage choice compresses it to 16 bits.
        solve(name="flop_3bet", board="Ks7s2d", pot=2000, stack=9000, storage="auto", iterations=6, check_every=3, **flop),
        # The flop of the benchmark in f32: the largest solve (20 GB of strategies).
        solve(name="flop_full", board="Ks7s2d", pot=600, stack=9700, iterations=4, check_every=4, **flop),
        # A session's river spots solved together.
        dict(name="batch_37", kind="batch", spots=37, plan=17, iterations=20, review=37),
        # The batched benchmark: 512 uneven river spots; some are opened for review.
        dict(name="batch_512", kind="batch", spots=512, plan=3000, iterations=50, review=16),
        # One data-parallel training step of the leaf network at the training batch.
        dict(name="net_train", kind="net", rows=256, hidden=1024, layers=4),
        # A flop cut at the turn deal, its leaves valued by the network.
        solve(name="flop_leafnet", kind="leafnet", board="Ks7s2d", pot=600, stack=9700, iterations=20, hidden=1024,
              layers=4, **flop),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def board(n):
        return "".join(abi.card_str(c) for c in rng.sample(range(52), n))

    def sizes():
        return ",".join(rng.sample(["33%", "50%", "75%", "100%", "150%"], rng.randint(1, 2)) + ["allin"])

    kind = rng.choice(["river"] * 6 + ["turn"] * 6 + ["flop"] * 4 + ["batch"] * 3 + ["net"] * 2 + ["leafnet"])
    if kind == "batch":
        n = log(1, 512)
        return dict(kind="batch", spots=n, plan=rng.randrange(1 << 20), iterations=log(5, 50), review=min(n, 16))
    if kind == "net":
        return dict(kind="net", rows=log(1, 1024), hidden=rng.choice([256, 512, 1024]), layers=rng.randint(2, 4))
    most = work(listed()[7])["bytes"]
    while True:
        ranges = rng.choice(["uniform", "dirichlet"])
        it = log(5, 100)
        c = solve(ranges=ranges, keep=log(12, 169), pot=log(300, 6000), stack=log(500, 15000), bets=sizes(),
                  raises=rng.choice(["2.5x", "3x"]), check_every=rng.choice([5, 10, 25]), iterations=it,
                  rake=rng.choice([0.0, 0.0, 0.05]))
        if kind == "river":
            c.update(board=board(5), precision=rng.choice(["fast"] * 4 + ["exact"]), keep_storage=rng.random() < 0.5)
        elif kind == "turn":
            c.update(board=board(4), precision=rng.choice(["fast"] * 5 + ["exact"]), keep_storage=rng.random() < 0.3,
                     storage=rng.choice(["f32", "f32", "compressed"]))
        elif kind == "flop":
            c.update(board=board(3), keep=log(12, 68), iterations=min(it, 40), storage=rng.choice(["f32", "auto"]))
            if rng.random() < 0.6:
                c.update(deal_turn=rng.randint(3, 12), deal_river=rng.randint(3, 12))
        else:
            c.update(kind="leafnet", board="Ks7s2d", ranges="dirichlet", keep=log(20, 68), rake=0.0, pot=600,
                     stack=log(1000, 9700), hidden=rng.choice([256, 512, 1024]), layers=rng.randint(2, 4))
        if c["precision"] == "exact":
            c["iterations"] = min(c["iterations"], 20 if kind == "river" else 3)
        if c["storage"] != "f32":
            c["keep_storage"] = False
        try:
            stats = Solver.estimate(config(c, 0))
        except Exception:
            continue
        if stats.total_nodes() < 3_000_000 and work(c)["bytes"] < most / 2:
            return c


# ------------------------------------------------------------------ inputs
def range_of(case, seed, p):
    """Player p's range: the hands in it come from the case, their weights from the seed."""
    f = workloads.expand_classes(1.0 - np.random.default_rng([seed, p]).random(169))
    if case["ranges"] == "uniform":
        return np.where(workloads.uniform_range(1000 + p, 169 - case["keep"]) > 0, f, np.float32(0.0))
    return workloads.dirichlet_range(2000 + p, case["keep"]) * np.maximum(f * f, np.float32(1e-4))


def config(case, seed):
    """The SolveConfig of a solve case."""
    ranges = [range_of(case, seed, p) for p in range(2)]
    sampled = (case["deal_turn"], case["deal_river"], 3) if case["deal_turn"] else None
    storage = {"f32": abi.STORAGE_F32, "auto": abi.STORAGE_AUTO, "compressed": abi.STORAGE_COMPRESSED}[case["storage"]]
    return abi.make_config(case["board"], ranges, pot=case["pot"], stack=case["stack"],
                           menu_=abi.menu(case["bets"].split(","), [case["raises"]]), storage=storage,
                           precision=case["precision"], sampled=sampled, rake_rate=case["rake"],
                           rake_cap=300.0 if case["rake"] else 0.0, max_memory_bytes=1 << 40, **workloads.DCFR)


def batch_specs(case):
    """(board, pot, stack, sizes) of each spot, from the case alone: uneven trees of 15 to 400 nodes."""
    rng = np.random.default_rng(case["plan"])
    zero = [np.ones(1326, np.float32)] * 2
    out = []
    while len(out) < case["spots"]:
        board = rng.choice(52, 5, replace=False).tolist()
        pot, stack = int(rng.integers(400, 6001)), int(rng.integers(2000, 15001))
        k = int(rng.integers(1, 4))
        sizes = [workloads.SIZES[i] for i in sorted(rng.choice(5, k, replace=False).tolist())] + ["allin"]
        est = Solver.estimate(abi.make_config(board, zero, pot=pot, stack=stack, menu_=abi.menu(sizes, sizes),
                                              storage=abi.STORAGE_F32, **workloads.DCFR))
        if 15 <= est.total_nodes() <= 400:
            out.append((board, pot, stack, sizes, est.storage_cells, est.total_nodes()))
    return out


def batch_range(seed, spot, p):
    return workloads.expand_classes(1.0 - np.random.default_rng([seed, spot, p]).random(169))


def pad128(x):
    return (x + 127) // 128 * 128


def net_shapes(case):
    dims = [IN_DIM] + [case["hidden"]] * case["layers"] + [OUT_DIM]
    return list(zip(dims[:-1], dims[1:]))


def net_params(case, seed):
    """Weights in the library's padded flat layout, and the same without padding."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    flat_w, flat_b, plain = [], [], []
    for k, n in net_shapes(case):
        w = torch.randn(n, k, device="cuda", generator=g) * (2.0 / k) ** 0.5
        b = torch.randn(n, device="cuda", generator=g) * 0.02
        full = torch.zeros(pad128(n), pad128(k), device="cuda")
        full[:n, :k] = w
        fb = torch.zeros(pad128(n), device="cuda")
        fb[:n] = b
        flat_w.append(full.reshape(-1))
        flat_b.append(fb)
        plain.append((w, b))
    return torch.cat(flat_w + flat_b), plain


def net_batch(case, seed):
    """Rows as the leaf data has them: two sparse ranges, one-hot cards, pot and stack; targets in pots."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = case["rows"]
    x = torch.zeros(m, IN_DIM, device="cuda")
    r = torch.rand(m, 2652, device="cuda", generator=g)
    x[:, :2652] = torch.where(r > 0.65, (r - 0.65) / 0.35, torch.zeros_like(r))
    x.scatter_(1, 2652 + torch.rand(m, 52, device="cuda", generator=g).argsort(1)[:, :4], 1.0)
    x[:, 2704:] = torch.rand(m, 2, device="cuda", generator=g)
    t = torch.randn(m, OUT_DIM, device="cuda", generator=g) * 0.3
    return x, t, (x[:, :2652] > 0).float()


def prepare(case, seed):
    if case["kind"] == "batch":
        cfgs = [abi.make_config(b, [batch_range(seed, i, 0), batch_range(seed, i, 1)], pot=pot, stack=stack,
                                menu_=abi.menu(sizes, sizes), storage=abi.STORAGE_F32, **workloads.DCFR)
                for i, (b, pot, stack, sizes, _, _) in enumerate(batch_specs(case))]
        b = BatchSolver.new(cfgs)
        b.autotune(10)
        return dict(case=case, batch=b)
    if case["kind"] == "net":
        net = LeafNet(IN_DIM, case["hidden"], case["layers"], OUT_DIM, max_batch=case["rows"], seed=0)
        net.set_params(net_params(case, seed)[0].cpu().numpy())
        return dict(case=case, net=net, data=net_batch(case, seed))
    cfg = config(case, seed)
    if case["kind"] == "leafnet":
        net = LeafNet(IN_DIM, case["hidden"], case["layers"], OUT_DIM, max_batch=49 * 32, seed=0)
        net.set_params(net_params(case, seed)[0].cpu().numpy())
        return dict(case=case, solver=Solver.new_depth_limited(cfg, net))
    s = Solver.new(cfg)
    keep = None
    if case["keep_storage"]:  # page-locked arrays that the program reads every solution into
        keep = tuple(torch.empty(s.storage_len(), dtype=torch.float32, pin_memory=True).numpy() for _ in range(2))
    return dict(case=case, solver=s, keep=keep)


# -------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.iterate(case["iterations"])
        e = b.exploitability()
        step = max(1, case["spots"] // case["review"])
        got = [b.download_storage(i) for i in range(0, case["spots"], step)]
        return dict(exploitability=e, regrets=np.concatenate([r for r, _ in got]), sums=np.concatenate([s for _, s in got]))
    if case["kind"] == "net":
        net = state["net"]
        loss = net.backward(*state["data"])
        net.adam_step(1e-3)
        gradients = net.grad_tensor()
        gradients.net = net  # a view of the network's buffer, valid while the network lives
        return dict(loss=loss, gradients=gradients)
    s = state["solver"]
    s.set_iterations(0)
    p = s.solve(SolveOptions(max_iterations=case["iterations"], target_exploitability_pct=0.0,
                             check_every=case["check_every"]))
    info = s.query(())
    out = dict(exploitability=p.exploitability, strategy=info.strategy, ev=info.ev, reach=info.reach)
    if state.get("keep"):
        out["regrets"], out["sums"] = s.download_storage(out=state["keep"])
    return out


# ------------------------------------------------------------------- work
def work(case):
    """Storage: 20 bytes a cell and iteration (10 in 16 bits): each regret read and written once, each regret and
    sum of the opponent read and the sum written; a check reads each sum once. Rows: one reach row read and one
    value row written per node and traversal. Terminals: about 12 operations per hand."""
    if case["kind"] == "net":
        m, macs = case["rows"], sum(k * n for k, n in net_shapes(case))
        # Forward and two backward products; weights and Adam's moments read and written, gradients written.
        return dict(bytes=32.0 * macs + 4.0 * m * (IN_DIM + 2 * OUT_DIM), flops=6.0 * m * macs)
    if case["kind"] == "batch":
        specs = batch_specs(case)
        cells, nodes = sum(x[4] for x in specs), sum(x[5] for x in specs)
        rows = 8.0 * nodes * 2 * 1081
        it = case["iterations"]
        return dict(bytes=it * (20.0 * cells + rows) + 4.0 * cells + rows, flops=(it + 1) * 14.0 * nodes * 1081)
    cfg = config(case, 0)
    cut = case["kind"] == "leafnet"
    if cut:
        # 16 decisions and their leaves: the network's products for 49 cards a leaf and traversal.
        it = case["iterations"] + case["iterations"] // case["check_every"]
        macs = sum(k * n for k, n in net_shapes(case))
        return dict(bytes=it * 2 * (2.0 * macs + 4.0 * 784 * (IN_DIM + OUT_DIM)), flops=it * 2 * 2.0 * 784 * macs)
    est = Solver.estimate(cfg)
    on = set(abi.parse_cards(case["board"]))
    free = np.array([not (set(abi.combo_cards(i)) & on) for i in range(1326)])
    n = [int(((np.array(cfg.ranges[p]) > 0) & free).sum()) for p in range(2)]
    it, checks = case["iterations"], max(1, case["iterations"] // case["check_every"])
    cell = 2.0 if est.compressed else 4.0
    rows = 8.0 * est.total_nodes() * (n[0] + n[1])
    passes = it + (checks * (2 if case["rake"] else 1) + 1)
    return dict(bytes=est.storage_cells * cell * (5 * it + checks + 1) + rows * passes +
                (8.0 * est.storage_cells if case["keep_storage"] else 0.0),
                flops=passes * 6.0 * est.terminal_nodes * (n[0] + n[1]) + 8.0 * it * est.storage_cells)


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """The same results in 64 bits from plain torch and numpy: river and turn games and the network."""
    if case["kind"] == "net":
        return exact_net(case, seed)
    if case["kind"] == "batch":
        if case["spots"] * case["iterations"] > 1500:
            return None
        step = max(1, case["spots"] // case["review"])
        e, regrets, sums = [], [], []
        for i, (b, pot, stack, sizes, _, _) in enumerate(batch_specs(case)):
            g = Game(b, [batch_range(seed, i, 0), batch_range(seed, i, 1)], pot, stack, sizes, sizes, 0.0)
            g.iterate(case["iterations"])
            e.append(g.exploitability())
            if i % step == 0:
                r, s = g.storage()
                regrets.append(r)
                sums.append(s)
        return dict(exploitability=np.array(e), regrets=np.concatenate(regrets), sums=np.concatenate(sums))
    cards = abi.parse_cards(case["board"])
    if case["kind"] == "leafnet" or len(cards) < 4 or case["storage"] != "f32":
        return None
    if len(cards) == 4 and case["iterations"] > 40:
        return None
    g = Game(cards, [range_of(case, seed, p) for p in range(2)], case["pot"], case["stack"],
             case["bets"].split(","), [case["raises"]], case["rake"])
    g.iterate(case["iterations"])
    strategy, ev, reach = g.root_query()
    out = dict(exploitability=torch.tensor(g.exploitability(), dtype=torch.float64), strategy=strategy, ev=ev, reach=reach)
    if case["keep_storage"]:
        out["regrets"], out["sums"] = g.storage() if len(cards) == 5 else (None, None)
    return out


def exact_net(case, seed):
    layers = [(w.double().requires_grad_(), b.double().requires_grad_()) for w, b in net_params(case, seed)[1]]
    x, t, mask = (v.double() for v in net_batch(case, seed))
    y = x
    for i, (w, b) in enumerate(layers):
        y = y @ w.T + b
        if i < len(layers) - 1:
            y = torch.nn.functional.gelu(y)
    loss = (mask * (y - t) ** 2).sum() / mask.sum()
    loss.backward()
    gw, gb = [], []
    for w, b in layers:
        n, k = w.shape
        full = torch.zeros(pad128(n), pad128(k), device="cuda", dtype=torch.float64)
        full[:n, :k] = w.grad
        fb = torch.zeros(pad128(n), device="cuda", dtype=torch.float64)
        fb[:n] = b.grad
        gw.append(full.reshape(-1))
        gb.append(fb)
    return dict(loss=loss.detach(), gradients=torch.cat(gw + gb))


HI = np.array([hi for hi in range(52) for lo in range(hi)])
LO = np.array([lo for hi in range(52) for lo in range(hi)])


def strengths(board, hi, lo):
    """Order of the hands' best five of seven cards: a whole number each."""
    cards = np.concatenate([np.tile(np.array(board), (len(hi), 1)), hi[:, None], lo[:, None]], 1)
    have = np.zeros((len(hi), 13, 4), bool)
    for k in range(7):
        have[np.arange(len(hi)), cards[:, k] // 4, cards[:, k] % 4] = True
    count = have.sum(2)

    def straight(m):  # highest rank of five in a row, -1: none
        w = np.concatenate([m[:, 12:], m], 1)
        best = np.full(len(m), -1)
        for top in range(3, 13):
            best = np.where(w[:, top - 3:top + 2].all(1), top, best)
        return best

    def top(m, k):  # the k highest set ranks as digits
        v, m = np.zeros(len(m), np.int64), m.copy()
        for _ in range(k):
            r = np.where(m.any(1), 12 - m[:, ::-1].argmax(1), -1)
            v = v * 14 + (r + 1)
            m[np.arange(len(m)), np.maximum(r, 0)] = False
        return v

    def one(m):
        return np.where(m.any(1), 12 - m[:, ::-1].argmax(1), -1)

    def without(m, r):
        m = m.copy()
        m[np.arange(len(m)), np.maximum(r, 0)] = False
        return m

    suited = have.transpose(0, 2, 1)
    flush = suited.sum(2) >= 5
    fm = suited[np.arange(len(hi)), flush.argmax(1)] & flush.any(1)[:, None]
    some = count > 0
    quad, trip, pair = one(count == 4), one(count == 3), one(count == 2)
    full = one(without(count >= 2, trip))
    second = one(without(count == 2, pair))
    sf, st = straight(fm), straight(some)
    score = top(some, 5)
    unit = 14 ** 5

    def put(ok, cat, low):
        nonlocal score
        score = np.where(ok, cat * unit + low, score)

    put(pair >= 0, 1, (pair + 1) * 14 ** 3 + top(without(some, pair), 3))
    put((pair >= 0) & (second >= 0), 2, ((pair + 1) * 14 + second + 1) * 14 + top(without(without(some, pair), second), 1))
    put(trip >= 0, 3, (trip + 1) * 14 ** 2 + top(without(some, trip), 2))
    put(st >= 0, 4, st + 1)
    put(flush.any(1), 5, top(fm, 5))
    put((trip >= 0) & (full >= 0), 6, (trip + 1) * 14 + full + 1)
    put(quad >= 0, 7, (quad + 1) * 14 + top(without(some, quad), 1))
    put(sf >= 0, 8, sf + 1)
    return score


class Game:
    """A heads-up river or turn game and its DCFR in 64 bits. Rows are [boards, hands]: one board on the root
    street of a turn game, 48 below the deal."""

    def __init__(self, cards, ranges, pot, stack, bets, raises, rake):
        self.pot, self.sizes, self.rake_rate = pot, (bets, raises), rake
        ok = ~np.isin(HI, cards) & ~np.isin(LO, cards)
        ids = [np.nonzero(ok & (np.asarray(r) > 0))[0] for r in ranges]
        hi, lo = [HI[i] for i in ids], [LO[i] for i in ids]
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.w = [torch.tensor(np.asarray(ranges[p])[ids[p]].astype(np.float64), device=dev)[None] for p in range(2)]
        deals = [[]] if len(cards) == 5 else [[c] for c in range(52) if c not in cards]
        self.river = len(cards) == 5
        self.deals = deals
        share = np.zeros((len(hi[0]), len(hi[1])), bool)
        for a in (hi[0], lo[0]):
            for b in (hi[1], lo[1]):
                share |= a[:, None] == b[None]
        fits = torch.tensor(~share, device=dev).double()
        self.fits = [fits, fits.T.contiguous()]
        self.free = [torch.tensor(np.array([~(np.isin(hi[p], d) | np.isin(lo[p], d)) for d in deals]), device=dev).double()
                     for p in range(2)]
        s = [torch.tensor(np.array([strengths(list(cards) + d, hi[p], lo[p]) for d in deals]), device=dev)
             for p in range(2)]
        m = fits[None] * self.free[0][:, :, None] * self.free[1][:, None, :]
        d = s[0][:, :, None] - s[1][:, None, :]
        self.win = [m * (d > 0), (m * (d < 0)).transpose(1, 2).contiguous()]
        self.lose = [m * (d < 0), (m * (d > 0)).transpose(1, 2).contiguous()]
        self.tie = [m * (d == 0), (m * (d == 0)).transpose(1, 2).contiguous()]
        self.norm = 1.0 / float(self.w[0][0] @ fits @ self.w[1][0])
        self.players = []
        st = dict(street=len(cards) - 2, pot=pot, commit=(0, 0), stack=(stack, stack), bet=0, inc=100, raises=0, act=0,
                  needs=(stack > 0, stack > 0))
        self.root = self.build(st, (0, 0))
        self.t = 0

    # The action tree: bets and raises rounded half up, clamped between the least raise and all-in.
    def actions(self, st):
        p, o = st["act"], 1 - st["act"]
        call = min(max(st["bet"] - st["commit"][p], 0), st["stack"][p])
        most = min(st["commit"][p] + st["stack"][p], st["commit"][o] + st["stack"][o])
        out = ["fold", "call"] if call > 0 else ["check"]
        if most <= st["bet"] or st["raises"] >= 3:
            return out
        to, least = set(), min(st["bet"] + max(st["inc"], 100), most)
        for s in self.sizes[1 if st["bet"] else 0]:
            if s == "allin":
                a = most
            elif s.endswith("%"):
                a = st["bet"] + math.floor(float(s[:-1]) / 100.0 * (st["pot"] + call) + 0.5)
            elif st["bet"] == 0:
                continue
            else:
                a = math.floor(float(s[:-1]) * st["bet"] + 0.5)
            to.add(min(max(a, least), most))
        return out + sorted(a for a in to if a > st["bet"])

    def build(self, st, inv):
        p, o = st["act"], 1 - st["act"]
        hands = self.w[p].shape[1]
        boards = 1 if st["street"] == 2 else len(self.deals)
        node = dict(kind="act", player=p, inv=inv, boards=boards, kids=[])
        acts = self.actions(st)
        node["r"] = torch.zeros(len(acts), boards, hands, dtype=torch.float64, device=self.w[0].device)
        node["s"] = torch.zeros_like(node["r"])
        self.players.append(node)
        for a in acts:
            s = dict(st)
            if a == "fold":
                left = max(st["commit"][o] - st["commit"][p], 0)
                node["kids"].append(dict(kind="fold", player=p, inv=inv, rake=self.rake(st["pot"] - left)))
                continue
            put = 0
            needs = list(st["needs"])
            if a == "call":
                put = min(max(st["bet"] - st["commit"][p], 0), st["stack"][p])
            elif a != "check":
                put = a - st["commit"][p]
                s["inc"] = max(st["inc"], a - st["bet"])
                s["bet"], s["raises"] = a, st["raises"] + 1
                needs[o] = st["stack"][o] > 0
            needs[p] = False
            s["commit"] = tuple(c + put * (i == p) for i, c in enumerate(st["commit"]))
            s["stack"] = tuple(c - put * (i == p) for i, c in enumerate(st["stack"]))
            s["pot"], s["needs"] = st["pot"] + put, tuple(needs)
            i2 = tuple(c + put * (i == p) for i, c in enumerate(inv))
            if needs[o]:
                s["act"] = o
                node["kids"].append(self.build(s, i2))
            else:
                node["kids"].append(self.over(s, i2))
        return node

    def over(self, st, inv):
        end = dict(kind="show", inv=inv, rake=self.rake(st["pot"]))
        if st["street"] == 3:
            return end
        if 0 in st["stack"]:
            return dict(kind="deal", kid=end)
        s = dict(street=3, pot=st["pot"], commit=(0, 0), stack=st["stack"], bet=0, inc=100, raises=0, act=0,
                 needs=(True, True))
        return dict(kind="deal", kid=self.build(s, inv))

    def rake(self, pot):
        return float(np.float32(min(pot * self.rake_rate, 300.0 if self.rake_rate else 0.0)))

    def sigma(self, x):
        d = x.sum(0)
        return torch.where(d > 0, x / torch.where(d > 0, d, torch.ones_like(d)), torch.full_like(x, 1.0 / len(x)))

    def value(self, node, p, reach, mode):
        """Counterfactual values [boards, hands] of player p under the opponent's reach."""
        o, half = 1 - p, self.pot / 2.0
        if node["kind"] == "fold":
            f, inv = node["player"], node["inv"]
            v = -(half + inv[p]) if f == p else half + inv[f] - node["rake"]
            return v * self.norm * (reach @ self.fits[p].T)
        if node["kind"] == "show":
            inv, rake = node["inv"], node["rake"]
            a, b, c = half + inv[o] - rake, -(half + inv[p]), 0.5 * (inv[o] - inv[p] - rake)
            col = reach[:, :, None]
            v = a * (self.win[p] @ col) + b * (self.lose[p] @ col)
            if c != 0.0:
                v = v + c * (self.tie[p] @ col)
            return self.norm * v[:, :, 0]
        if node["kind"] == "deal":
            v = self.value(node["kid"], p, reach * self.free[o] / 44.0, mode)
            return (v * self.free[p]).sum(0, keepdim=True)
        live = (reach != 0).any(1)[None, :, None]
        if node["player"] == o:
            x = node["r"].clamp(min=0) if mode == "cfr" else node["s"]
            sig = self.sigma(x)
            if mode == "cfr":
                node["s"] = torch.where(live, node["s"] * self.disc[2] + sig, node["s"])
            return sum(self.value(k, p, reach * sig[a], mode) for a, k in enumerate(node["kids"]))
        vals = torch.stack([self.value(k, p, reach, mode) for k in node["kids"]])
        if mode == "br":
            return vals.max(0).values
        if mode == "avg":
            return (self.sigma(node["s"]) * vals).sum(0)
        r = node["r"]
        v = (self.sigma(r.clamp(min=0)) * vals).sum(0)
        node["r"] = torch.where(live, r * torch.where(r > 0, self.disc[0], self.disc[1]) + vals - v, r)
        return v

    def iterate(self, n):
        for _ in range(n):
            self.t += 1
            prev = float(self.t - 1)
            since = prev - (4.0 ** math.floor(math.log(prev, 4) + 1e-12) if prev else 0.0)
            self.disc = (prev ** 1.5 / (prev ** 1.5 + 1.0), 0.5, (since / (since + 1.0)) ** 2)
            for p in range(2):
                self.value(self.root, p, self.w[1 - p], "cfr")

    def total(self, mode):
        return [float((self.value(self.root, p, self.w[1 - p], mode) * self.w[p]).sum()) for p in range(2)]

    def exploitability(self):
        v = sum(self.total("br"))
        return (v - sum(self.total("avg"))) / 2.0 if self.rake_rate else v / 2.0

    def root_query(self):
        reach = self.w[1]
        mass = (reach @ self.fits[0].T) * self.norm
        ev = torch.stack([self.value(k, 0, reach, "avg") for k in self.root["kids"]])[:, 0]
        ev = torch.where(mass > 0, ev / torch.where(mass > 0, mass, torch.ones_like(mass)) + self.pot / 2.0,
                         torch.zeros_like(mass))
        return self.sigma(self.root["s"])[:, 0].cpu(), ev.cpu(), self.w[0][0].cpu()

    def storage(self):
        """Regrets and strategy sums in the library's node order."""
        return tuple(np.concatenate([n[k].reshape(-1).cpu().numpy() for n in self.players]) for k in ("r", "s"))

"""The calls this library's users make, as cases that can be timed and compared.

Each kind of case below goes through the package's public entry points over
the range of sizes and options that its workloads, drivers and tests use:

* eval7        7-card evaluation: a handful of hands up to bulk scoring
* counts       showdown win/tie/loss counts of a board (flop, turn, river)
* dump         the flop-EV dump, for some flops or for all 1,755
* river_spot   one river subgame, host data in, strategies and values out
* river_batch  many uneven river subgames resident on the device
* turn         a heads-up turn + river tree (chance layer of river cards)
* diff_ev      differentiable EV, forward and backward through autograd
* multiway     the four-player ICM river
* leaf_rows    inference of the leaf network
* leaf_train   an epoch of training steps of the leaf network
* preflop      the preflop anchor chain (all-in matrix, flop matrices, DCFR)

`listed` names the cases, `draw` gives more of the same ranges, `prepare`
makes a case's inputs and handles from a seed, `run` is one pass, `work` the
bytes and operations the pass cannot do without and `exact` the 64-bit values
of its outputs in plain torch and numpy.
"""
import importlib
import math

import numpy as np
import torch

mtt = importlib.import_module("mtt-gpu-solver_b200")
wl = importlib.import_module("mtt-gpu-solver_b200.workloads")
mw = importlib.import_module("mtt-gpu-solver_b200.multiway")
dv = importlib.import_module("mtt-gpu-solver_b200.diffev")
ln = importlib.import_module("mtt-gpu-solver_b200.leafnet")
pf = importlib.import_module("mtt-gpu-solver_b200.preflop")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a few hands scored between other work (a range editor, a unit of a simulation)
        {"name": "eval7_few", "kind": "eval7", "n": 1009},
        # bulk scoring of sampled hands
        {"name": "eval7_bulk", "kind": "eval7", "n": 30_000_001},
        # the turn equity counts of every pair of live combos
        {"name": "turn_counts", "kind": "counts", "nboard": 4, "hands": 1128},
        # the whole flop-EV dump (the ev_dumper program)
        {"name": "flop_dump", "kind": "dump", "n": 1755},
        # one river spot solved from host data (the hu_solver program, an interactive tool)
        {"name": "river_spot", "kind": "river_spot", "hands": 1081, "pot": 100.0, "stack": 200.0, "sizes": "0.5,1.0",
         "cap": 1, "iters": 1000, "algo": 0, "semantics": 0, "alternate": True, "avg_power": 2.0},
        # a batch of uneven subgames solved for their root values (training data, range studies)
        {"name": "river_batch", "kind": "river_batch", "n": 1024, "max_sizes": 4, "iters": 200},
        # a deep turn spot with the river dealt (DCFR): the values and best responses of every hand
        {"name": "turn_dcfr", "kind": "turn", "hands": 1128, "pot": 60.0, "stack": 470.0, "sizes": "0.33,0.75,1.5",
         "cap": 2, "iters": 50, "algo": 1},
        # gradients of the EV with respect to both ranges and all strategy logits
        {"name": "diff_ev", "kind": "diff_ev", "n": 1024, "hands": 1081},
        # the four-player ICM river (the multiway_solver program)
        {"name": "multiway", "kind": "multiway", "hands": 1081, "cap": 2, "iters": 100, "semantics": 0, "algo": 0},
        # the network's rows of five turn leaves: 48 river cards each
        {"name": "leaf_rows", "kind": "leaf_rows", "rows": 240},
        # one epoch of 12,288 samples at the training loop's batch size
        {"name": "leaf_train", "kind": "leaf_train", "batch": 512, "steps": 24, "weights": True},
        # the preflop chain over a 100-flop subset (the preflop_gen program)
        {"name": "preflop", "kind": "preflop", "flops": 100, "iters": 500, "mode": 0},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval7", "counts", "dump", "river_spot", "river_batch", "turn", "diff_ev", "multiway",
                       "leaf_rows", "leaf_train", "preflop"])
    c = {"kind": kind}
    if kind == "eval7":
        c["n"] = _logint(rng, 500, 30_000_001)
    elif kind == "counts":
        c["nboard"] = rng.choice([3, 4, 5])
        c["hands"] = rng.randint(100, {3: 1176, 4: 1128, 5: 1081}[c["nboard"]])
    elif kind == "dump":
        c["n"] = _logint(rng, 1, 1755)
    elif kind == "river_spot":
        c.update(hands=rng.randint(200, 1081), pot=round(rng.uniform(20.0, 200.0), 1),
                 sizes=rng.choice(["0.5,1.0", "0.75", "0.33,0.8", "1.0"]), cap=rng.randint(1, 2),
                 iters=rng.randint(200, 1000), algo=rng.choice([0, 0, 1]), semantics=rng.choice([0, 0, 1]),
                 alternate=rng.choice([True, True, False]), avg_power=rng.choice([1.0, 2.0]))
        c["stack"] = round(c["pot"] * rng.uniform(0.5, 4.0), 1)
    elif kind == "river_batch":
        c.update(n=_logint(rng, 12, 1024), max_sizes=rng.randint(1, 4), iters=rng.randint(50, 200))
    elif kind == "turn":
        c.update(hands=rng.randint(300, 1128), pot=round(rng.uniform(20.0, 200.0), 1),
                 sizes=rng.choice(["0.5", "0.5,1.0", "0.33,0.75"]), cap=1, iters=rng.randint(10, 50),
                 algo=rng.choice([0, 1]))
        c["stack"] = round(c["pot"] * rng.uniform(1.0, 6.0), 1)
    elif kind == "diff_ev":
        c.update(n=_logint(rng, 8, 1024), hands=rng.randint(200, 1081))
    elif kind == "multiway":
        c.update(hands=rng.randint(200, 1081), cap=rng.randint(1, 2), iters=rng.randint(20, 100),
                 semantics=rng.choice([0, 0, 1]), algo=rng.choice([0, 0, 1]))
    elif kind == "leaf_rows":
        c["rows"] = _logint(rng, 48, 4096)
    elif kind == "leaf_train":
        c.update(batch=8 * _logint(rng, 8, 128), steps=rng.randint(4, 12), weights=rng.choice([True, False]))
    else:
        c.update(flops=_logint(rng, 4, 100), iters=rng.randint(50, 500), mode=rng.choice([0, 1]))
    return c


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    return torch.Generator(device=_dev()).manual_seed(seed)


_PAIRS = np.array([(a, b) for a in range(52) for b in range(a + 1, 52)], np.int64)


def _live(board):
    return np.nonzero(~np.isin(_PAIRS, np.asarray(board)).any(axis=1))[0].astype(np.uint16)


def _support(rng, board, k):
    live = _live(board)
    return live if k >= len(live) else np.sort(rng.choice(live, size=k, replace=False)).astype(np.uint16)


def _sizes(case):
    return [float(s) for s in case["sizes"].split(",")]


def _spot(case, seed, street):
    """A seeded river (5) or turn (4) subgame; Dirichlet(0.3) ranges."""
    rng = np.random.default_rng(seed)
    board = [int(x) for x in rng.choice(52, size=street, replace=False)]
    nodes, rows, _ = mtt.build_tree(case["pot"], case["stack"], _sizes(case), raise_cap=case["cap"], street=street,
                                    board=board if street == 4 else None)
    g = {"nodes": nodes, "rows": rows, "board": board, "pot": case["pot"]}
    for p in (0, 1):
        c = _support(rng, board, case["hands"])
        w = rng.dirichlet(np.full(len(c), 0.3))
        g[f"combos{p}"], g[f"range{p}"] = c, (w / w.sum()).astype(np.float32)
    return g


def _cfr_params(case):
    if case["kind"] == "turn":
        return mtt.solve_params(iters=case["iters"], algo=case["algo"], exploitability=True, avg_power=2.0)
    return mtt.solve_params(iters=case["iters"], algo=case["algo"], semantics=case["semantics"], exploitability=True,
                            alternate=case["alternate"], avg_power=case["avg_power"])


def _river_batch(case, seed):
    """Uneven subgames: trees and support sizes of the seeded batch workload, boards, supports and weights from seed."""
    rng = np.random.default_rng(seed)
    subs = wl.river_batch(n=case["n"], seed=2, max_sizes=case["max_sizes"])
    for g in subs:
        g["board"] = [int(x) for x in rng.choice(52, size=5, replace=False)]
        for p in (0, 1):
            c = _support(rng, g["board"], len(g[f"combos{p}"]))
            g[f"combos{p}"], g[f"range{p}"] = c, rng.lognormal(0.0, 1.0, size=len(c)).astype(np.float32)
    return subs


def _multiway_sub(case, seed):
    """The ICM workload's seats, stacks and tree; board, combos and ranges from seed."""
    rng = np.random.default_rng(seed)
    g = wl.multiway_icm(seed=4, n_hands=2, raise_cap=case["cap"])
    g["board"] = [int(x) for x in rng.choice(52, size=5, replace=False)]
    g["combos"] = _support(rng, g["board"], case["hands"])
    w = [rng.dirichlet(np.full(len(g["combos"]), 0.3)) for _ in range(4)]
    g["ranges"] = [(r / r.sum()).astype(np.float32) for r in w]
    return g


def _hands7(n, seed):
    """n uniform 7-card hands (distinct cards), uint8 [n, 7]."""
    g, out = _gen(seed), []
    for i in range(0, n, 2_000_000):
        m = min(2_000_000, n - i)
        out.append(torch.rand((m, 52), device=_dev(), generator=g).topk(7, dim=1).indices.to(torch.uint8))
    return torch.cat(out)


def _counts_inputs(case, seed):
    rng = np.random.default_rng(seed)
    board = rng.choice(52, size=case["nboard"], replace=False).astype(np.uint8)
    return board, _PAIRS[_support(rng, board, case["hands"])].astype(np.uint8)


def _flops(n, seed):
    """n of the 1,755 canonical flops, shuffled, and their orbit weights."""
    meta = mtt.canonical_flops()
    meta = meta[np.random.default_rng(seed).choice(len(meta), size=n, replace=False)]
    return np.ascontiguousarray(meta[:, :3]), meta[:, 3].astype(np.float32)


def _leaf_features(n, seed):
    """Feature rows as the training sets hold them, and the live combos of each row."""
    g, d = _gen(seed), _dev()
    board = torch.rand((n, 52), device=d, generator=g).topk(5, dim=1).indices
    onb = torch.zeros((n, 52), device=d).scatter_(1, board, 1.0)
    pairs = torch.as_tensor(_PAIRS, device=d)
    live = (onb[:, pairs[:, 0]] + onb[:, pairs[:, 1]]) == 0
    x = torch.zeros((n, ln.IN), device=d)
    for p in (0, 1):
        w = torch.exp(1.5 * torch.randn((n, 1326), device=d, generator=g)) * live
        x[:, p * 1326:(p + 1) * 1326] = w / w.sum(1, keepdim=True) * 1081.0
    x[:, 2652:2704] = onb
    x[:, 2704] = 1.0
    x[:, 2705] = 0.5 + 3.5 * torch.rand(n, device=d, generator=g)
    return x, live


def _leaf_train_inputs(case, seed):
    n = case["batch"] * case["steps"]
    x, live = _leaf_features(n, seed)
    w = torch.cat([live, live], 1).float()
    t = 0.1 * torch.randn((n, ln.OUT), device=x.device, generator=_gen(seed + 1)) * w
    return x, t, w if case["weights"] else None


def _diff_inputs(case, seed):
    """n river boards with one betting tree: full [n, 1326] ranges, N(0, 1) logits in the packed rows layout."""
    rng = np.random.default_rng(seed)
    nodes, rows, _ = mtt.build_tree(100.0, 200.0, [0.5, 1.0], raise_cap=1)
    subs, combos = [], []
    for _ in range(case["n"]):
        board = [int(x) for x in rng.choice(52, size=5, replace=False)]
        c = _support(rng, board, case["hands"])
        r = np.full(len(c), 1.0 / len(c), np.float32)
        subs.append({"nodes": nodes, "rows": rows, "board": board, "combos0": c, "combos1": c, "range0": r,
                     "range1": r, "pot": 100.0})
        combos.append(c.astype(np.int64))
    H = len(combos[0])
    Hp = (H + 3) // 4 * 4
    g, d = _gen(seed), _dev()
    logits = torch.randn((case["n"], int(rows[0]) + int(rows[1]), Hp), device=d, generator=g)
    logits[:, :, H:] = 0.0
    full = []
    sel = torch.as_tensor(np.stack(combos), device=d)
    for _ in (0, 1):
        w = torch.rand((case["n"], H), device=d, generator=g)
        full.append(torch.zeros((case["n"], 1326), device=d).scatter_(1, sel, w / w.sum(1, keepdim=True)))
    return subs, sel, logits, full[0], full[1]


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    k = case["kind"]
    st = {"case": case}
    if k == "eval7":
        st["cards"] = _hands7(case["n"], seed)
    elif k == "counts":
        board, hands = _counts_inputs(case, seed)
        st["board"], st["hands"] = torch.from_numpy(board).cuda(), torch.from_numpy(hands).cuda()
    elif k == "dump":
        st["flops"] = torch.from_numpy(_flops(case["n"], seed)[0]).cuda()
    elif k == "river_spot":
        st["sub"], st["params"] = _spot(case, seed, 5), _cfr_params(case)
    elif k == "river_batch":
        st["batch"] = mtt.RiverBatch(_river_batch(case, seed))
        st["params"] = mtt.solve_params(iters=case["iters"], exploitability=True, avg_power=2.0)
    elif k == "turn":
        st["batch"], st["params"] = mtt.RiverBatch([_spot(case, seed, 4)]), _cfr_params(case)
    elif k == "diff_ev":
        subs, _, logits, r0, r1 = _diff_inputs(case, seed)
        st["ev"] = dv.StrategyEV(subs)
        st["logits"] = logits.reshape(-1).requires_grad_()
        st["r0"], st["r1"] = r0.requires_grad_(), r1.requires_grad_()
    elif k == "multiway":
        st["batch"] = mw.MultiwayBatch([_multiway_sub(case, seed)])
        st["params"] = mtt.solve_params(iters=case["iters"], semantics=case["semantics"], algo=case["algo"])
    elif k == "leaf_rows":
        st["net"] = ln.LeafNet(batch_cap=(case["rows"] + 7) // 8 * 8, seed=seed)
        st["x"] = _leaf_features(case["rows"], seed)[0]
    elif k == "leaf_train":
        st["net"] = ln.LeafNet(batch_cap=case["batch"], seed=seed)
        st["x"], st["t"], st["w"] = _leaf_train_inputs(case, seed)
    else:
        st["flops"], st["weights"] = _flops(case["flops"], seed)
    return st


def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "eval7":
        return mtt.eval7(st["cards"])
    if k == "counts":
        return mtt.board_showdown_counts(st["board"], st["hands"])
    if k == "dump":
        return mtt.ev_dump(st["flops"])
    if k == "river_spot":
        b = mtt.RiverBatch([st["sub"]])
        b.solve(st["params"], graph=True)
        out = dict(b.read(0), results=b.results())
        b.close()
        return out
    if k == "river_batch":
        b = st["batch"]
        b.solve(st["params"], graph=True)
        vals = [b.root_values(s) for s in range(b.n)]
        return [b.results()] + [np.concatenate([v[i] for v in vals]) for i in range(4)]
    if k == "turn":
        b = st["batch"]
        b.solve(st["params"], graph=True)
        return (b.results(),) + b.root_values(0)
    if k == "diff_ev":
        logits, r0, r1, ev = st["logits"], st["r0"], st["r1"], st["ev"]
        logits.grad = r0.grad = r1.grad = None
        v = ev(logits, ev.pack_ranges(r0, r1))
        v.sum().backward()
        return v.detach(), logits.grad, r0.grad, r1.grad
    if k == "multiway":
        b = st["batch"]
        b.solve(st["params"], graph=True)
        return dict(b.read(0), values=b.values())
    if k == "leaf_rows":
        return st["net"].forward(st["x"])
    if k == "leaf_train":
        net, x, t, w, m = st["net"], st["x"], st["t"], st["w"], case["batch"]
        for i in range(0, len(x), m):
            net.train_step(x[i:i + m], t[i:i + m], None if w is None else w[i:i + m], lr=1e-4, want_loss=False)
        return [net.params(layer) for layer in range(4)]
    allin = pf.allin_matrix(case["mode"])
    mats = pf.flop_class_matrices(st["flops"], case["mode"])
    sums, sigma = pf.dcfr(st["weights"], mats, allin, iters=case["iters"])
    return allin, mats, sums, sigma


# ------------------------------------------------------------------ necessary work
# A hand's score takes about 60 integer operations, a compare of two scores one
# (win and tie counts: two).
def _tree_work(nodes, rows, hands, iters, passes, players):
    """Bytes: regrets and strategy sums in and out once per solve.  Operations per iteration: an update of every
    regret row and hand (about 12), and per terminal and player about 16 per hand for its value, each pass."""
    n_term = int(np.count_nonzero((nodes["type"] == 1) | (nodes["type"] == 2)))
    r = float(np.sum(rows)) * hands
    return {"bytes": 16.0 * r, "flops": iters * (12.0 * r + 16.0 * n_term * hands * players + 4.0 * r * (passes - 1))}


def work(case):
    k = case["kind"]
    if k == "eval7":
        return {"bytes": 11.0 * case["n"], "flops": 60.0 * case["n"]}
    if k == "counts":
        h, nb = case["hands"], case["nboard"]
        comp = {3: 1176, 4: 48, 5: 1}[nb]
        return {"bytes": 12.0 * h * h + 2 * h + nb, "flops": comp * (60.0 * h + 2.0 * h * h / 2)}
    if k == "dump":
        return {"bytes": case["n"] * (3.0 + 1352 * 4), "flops": case["n"] * 192.0 * (60.0 * 1176 + 2.0 * 1176 * 294)}
    if k in ("river_spot", "turn"):
        g = _spot(case, 0, 5 if k == "river_spot" else 4)
        h = min(case["hands"], {"river_spot": 1081, "turn": 1128}[k])
        return _tree_work(g["nodes"], g["rows"], h, case["iters"], 2, 2)
    if k == "river_batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for g in wl.river_batch(n=min(case["n"], 64), seed=0, max_sizes=case["max_sizes"]):
            h = 0.5 * (len(g["combos0"]) + len(g["combos1"]))
            w = _tree_work(g["nodes"], g["rows"], h, case["iters"], 2, 2)
            for key in tot:
                tot[key] += w[key] * case["n"] / min(case["n"], 64)
        return tot
    if k == "diff_ev":
        nodes, rows, _ = mtt.build_tree(100.0, 200.0, [0.5, 1.0], raise_cap=1)
        r = float(sum(rows)) * case["hands"] * case["n"]
        t = int(np.count_nonzero((nodes["type"] == 1) | (nodes["type"] == 2)))
        return {"bytes": 8.0 * r + case["n"] * 1326 * 16.0, "flops": 16.0 * r + 32.0 * t * case["hands"] * case["n"]}
    if k == "multiway":
        g = _multiway_sub(case, 4)
        return _tree_work(g["nodes"], g["rows"], case["hands"], case["iters"], 1, 4)
    weights = ln.IN * ln.HIDDEN + 2 * ln.HIDDEN * ln.HIDDEN + ln.HIDDEN * ln.OUT
    if k == "leaf_rows":
        return {"bytes": 2.0 * weights + 4.0 * case["rows"] * (ln.IN + ln.OUT), "flops": 2.0 * weights * case["rows"]}
    if k == "leaf_train":
        rows = case["batch"] * case["steps"]
        per_row = ln.IN + ln.OUT * (2 if case["weights"] else 1)
        return {"bytes": 4.0 * rows * per_row + 28.0 * weights * case["steps"],
                "flops": (6.0 * weights - 2.0 * ln.IN * ln.HIDDEN) * rows}
    n, combos = case["flops"], 1176 if case["mode"] == 0 else 1326
    return {"bytes": 4.0 * n * 169 * 169, "flops": 28561.0 * 3000 * 120 + n * (1176 * combos * 60.0 +
            2.0 * 190 * combos * combos) + 8.0 * case["iters"] * n * 169 * 169}


# ------------------------------------------------------------------ 64-bit values
def _tables():
    """Per 13-bit rank mask: highest rank (-1 if none), top rank of a straight (-1 if none), number of ranks, the
    mask of its five highest ranks."""
    hi, st, cnt, top = (np.full(8192, -1, np.int64) for _ in range(4))
    for m in range(8192):
        bits = [r for r in range(13) if m >> r & 1]
        hi[m] = bits[-1] if bits else -1
        cnt[m] = len(bits)
        top[m] = sum(1 << r for r in bits[-5:])
        run = [r for r in range(4, 13) if m >> (r - 4) & 31 == 31]
        st[m] = run[-1] if run else (3 if m & 0x100F == 0x100F else -1)
    return [torch.as_tensor(t, device=_dev()) for t in (hi, st, cnt, top)]


def _rank(cards, tabs):
    """Strength of 7 cards each (list of 7 broadcastable int64 tensors): larger wins, equal ties.  Quads, trips and
    pairs count a rank seen exactly 4, 3 and 2 times and compare without kickers; a suit flushes on 5 cards."""
    hi, st, _, top = tabs
    one = two = three = four = five = torch.zeros((), dtype=torch.int64, device=hi.device)
    sm, sc = [one] * 4, [one] * 4
    for c in cards:
        b = torch.ones_like(c) << (c >> 2)
        five, four, three, two, one = five | (four & b), four | (three & b), three | (two & b), two | (one & b), one | b
        for s in range(4):
            on = ((c & 3) == s).long()
            sm[s], sc[s] = sm[s] | (b * on), sc[s] + on
    quads, trips, pairs = four & ~five, three & ~four, two & ~three
    cat = lambda n, v: (n << 16) + v
    t1, p1 = hi[trips], hi[pairs]
    t2 = hi[trips & ~(1 << t1.clamp(min=0))]
    p2 = hi[pairs & ~(1 << p1.clamp(min=0))]
    straight = st[one]
    out = one
    out = torch.where(p1 >= 0, cat(1, p1), out)
    out = torch.where((p1 >= 0) & (p2 >= 0), cat(2, (p1 << 4) + p2), out)
    out = torch.where(t1 >= 0, cat(3, t1), out)
    out = torch.where(straight >= 0, cat(4, straight), out)
    out = torch.where((t1 >= 0) & ((t2 >= 0) | (p1 >= 0)), cat(6, (t1 << 4) + torch.where(t2 >= 0, t2, p1)), out)
    out = torch.where(quads > 0, cat(7, hi[quads]), out)
    for s in range(4):
        sf = st[sm[s]]
        out = torch.where(sc[s] >= 5, torch.where(sf >= 0, cat(8, sf), cat(5, top[sm[s]])), out)
    return out


def _ints(a):
    return torch.as_tensor(np.asarray(a, dtype=np.int64), device=_dev())


def _board_rank(board, combos, tabs):
    pr = _ints(_PAIRS[np.asarray(combos, np.int64)])
    return _rank([_ints(int(c)) for c in board] + [pr[:, 0], pr[:, 1]], tabs)


def _disjoint(ca, cb):
    """[len(ca), len(cb)] 1.0 where the two combos share no card."""
    a, b = _ints(_PAIRS[np.asarray(ca, np.int64)]), _ints(_PAIRS[np.asarray(cb, np.int64)])
    eq = torch.zeros((len(a), len(b)), dtype=torch.bool, device=a.device)
    for i in (0, 1):
        for j in (0, 1):
            eq |= a[:, i, None] == b[None, :, j]
    return (~eq).double()


def _groups(mask, *keys):
    """Index arrays of the nodes in mask, split by equal keys."""
    idx = np.nonzero(mask)[0]
    if len(idx) == 0:
        return []
    key = np.stack([np.asarray(k)[idx] for k in keys], 1)
    u, inv = np.unique(key, axis=0, return_inverse=True)
    return [(tuple(int(x) for x in u[i]), idx[inv.reshape(-1) == i]) for i in range(len(u))]


class _HeadsUp:
    """A heads-up river or turn subgame in float64, level by level."""

    def __init__(self, g, semantics):
        nd = g["nodes"]
        n = len(nd)
        d = _dev()
        self.n, self.nd, self.sem = n, nd, semantics
        self.combos = [g["combos0"], g["combos1"]]
        self.H = [len(c) for c in self.combos]
        self.rows = [int(r) for r in g["rows"]]
        self.range = [torch.as_tensor(np.asarray(g[f"range{p}"], np.float64), device=d) for p in (0, 1)]
        depth, dealt = np.zeros(n, np.int64), np.full(n, -1, np.int64)
        for i in range(n):
            if nd["type"][i] in (0, 3):
                ch = np.arange(nd["num_actions"][i]) + nd["children_offset"][i]
                depth[ch] = depth[i] + 1
                dealt[ch] = nd["turn_idx"][ch] if nd["type"][i] == 3 else dealt[i]
        self.levels = []
        for k in range(int(depth.max()) + 1):
            at = depth == k
            dec = [(p, A, _ints(i), _ints(nd["children_offset"][i])[:, None] + torch.arange(A, device=d),
                    _ints(nd["infoset_offset"][i])[:, None] + torch.arange(A, device=d))
                   for (p, A), i in _groups(at & (nd["type"] == 0), nd["player"], nd["num_actions"])]
            deal = [(int(i), int(nd["num_actions"][i]), int(nd["children_offset"][i]))
                    for i in np.nonzero(at & (nd["type"] == 3))[0]]
            self.levels.append((dec, deal))
        tabs = _tables()
        self.C = _disjoint(*self.combos)                       # [H0, H1]
        col = lambda x: torch.as_tensor(np.asarray(x, np.float64), device=d)[:, None]
        pr = [_ints(_PAIRS[np.asarray(c, np.int64)]) for c in self.combos]
        free = lambda p, card: ((pr[p][:, 0] != card) & (pr[p][:, 1] != card)).double()
        self.free = {int(c): [free(0, int(c)), free(1, int(c))] for c in np.unique(dealt)}
        self.folds, self.shows = [], []
        for (c,), i in _groups(nd["type"] == 1, dealt):
            win = np.where(nd["active_mask"][i] == 1, 0, 1)
            pay = [col(np.where(win == q, nd["pot_size"][i].astype(np.float64), 0.0) - nd["committed"][i, q])
                   for q in (0, 1)]
            self.folds.append((c, _ints(i), pay))
        for (c,), i in _groups(nd["type"] == 2, dealt):
            s = [_board_rank(list(g["board"]) + ([c] if c >= 0 else []), x, tabs) for x in self.combos]
            a, b = s[0][:, None], s[1][None, :]
            A0 = ((a > b).double() + 0.5 * (a == b).double()) * self.C          # share of player 0, [H0, H1]
            self.shows.append((c, _ints(i), col(nd["pot_size"][i]), [col(nd["committed"][i, q]) for q in (0, 1)], A0))
        self.n_live = 52 - len(g["board"])

    def terminals(self, reach, q, v, sem):
        ro, C = reach[1 - q], self.C.T if q == 0 else self.C                    # C: [opponent, own]
        for c, i, pay in self.folds:
            r = ro[i]
            v[i] = pay[q] * (r @ C if sem == 0 else r.sum(1, keepdim=True)) * self.free[c][q]
        for c, i, pot, com, A0 in self.shows:
            r = ro[i]
            A = A0.T if q == 0 else self.C - A0
            if sem == 0:
                v[i] = (pot * (r @ A) - com[q] * (r @ C)) * self.free[c][q]
            else:
                tot = r.sum(1, keepdim=True)
                v[i] = pot * (r @ A if q == 0 else tot - r @ A) - com[q] * tot

    def down(self, reach, policy):
        for p in (0, 1):
            reach[p][0] = self.range[p]
        for dec, deal in self.levels:
            for p, A, i, ch, row in dec:
                reach[p][ch] = reach[p][i][:, None] * policy[p][row]
                reach[1 - p][ch] = reach[1 - p][i][:, None].expand(-1, A, -1)
            for i, A, first in deal:
                for a in range(A):
                    f = self.free[int(self.nd["turn_idx"][first + a])]
                    for p in (0, 1):
                        reach[p][first + a] = reach[p][i] * f[p]

    def up_chance(self, deal, v, q, sem):
        for i, A, first in deal:
            v[i] = 0.0
            for a in range(A):
                v[i] += v[first + a] * self.free[int(self.nd["turn_idx"][first + a])][q]
            v[i] /= self.n_live - (2 if sem else 4)

    def normalise(self, X, p, floor):
        out = torch.zeros_like(X)
        for dec, _ in self.levels:
            for q, A, _, _, row in dec:
                if q == p:
                    pos = X[row].clamp(min=0.0)
                    s = pos.sum(1, keepdim=True)
                    out[row] = torch.where(s > floor, pos / torch.where(s > floor, s, torch.ones_like(s)),
                                           torch.full_like(pos, 1.0 / A))
        return out

    def solve(self, iters, algo, alternate, avg_power, alpha=1.5, beta=0.0, gamma=2.0):
        z = lambda m, p: torch.zeros((m, self.H[p]), dtype=torch.float64, device=_dev())
        R, S = [z(self.rows[p], p) for p in (0, 1)], [z(self.rows[p], p) for p in (0, 1)]
        reach, cfv = [z(self.n, p) for p in (0, 1)], [z(self.n, p) for p in (0, 1)]
        sig = [self.normalise(R[p], p, 1e-7) for p in (0, 1)]
        for t in range(1, iters + 1):
            w = float(t) ** avg_power
            dpos, dneg = ((t - 1.0) ** e / ((t - 1.0) ** e + 1.0) for e in (alpha, beta))
            dstr = ((t - 1.0) / t) ** gamma
            for upd in ([(0,), (1,)] if alternate else [(0, 1)]):
                self.down(reach, sig)
                for p in upd:
                    if algo:
                        S[p] *= dstr
                    for dec, _ in self.levels:
                        for q, A, i, ch, row in dec:
                            if q == p:
                                S[p][row] += reach[p][i][:, None] * sig[p][row] * (1.0 if algo else w)
                    v = cfv[p]
                    self.terminals(reach, p, v, self.sem)
                    for dec, deal in reversed(self.levels):
                        for q, A, i, ch, row in dec:
                            if q != p:
                                v[i] = v[ch].sum(1)
                                continue
                            val = (sig[p][row] * v[ch]).sum(1)
                            v[i] = val
                            inst = v[ch] - val[:, None]
                            r = R[p][row]
                            R[p][row] = r * torch.where(r > 0, dpos, dneg) + inst if algo else (r + inst).clamp(min=0)
                        self.up_chance(deal, v, p, self.sem)
                for p in upd:
                    sig[p] = self.normalise(R[p], p, 1e-7)
        return R, S, [cfv[p][0].clone() for p in (0, 1)]

    def values(self, S):
        """The average strategies' results row and both players' root values and best-response values."""
        pol = [self.normalise(S[p], p, 0.0) for p in (0, 1)]
        z = lambda p: torch.zeros((self.n, self.H[p]), dtype=torch.float64, device=_dev())
        reach = [z(0), z(1)]
        self.down(reach, pol)
        ev, br, root = [], [], []
        for p in (0, 1):
            v, b = z(p), z(p)
            self.terminals(reach, p, v, 0)
            self.terminals(reach, p, b, 0)
            for dec, deal in reversed(self.levels):
                for q, A, i, ch, row in dec:
                    v[i] = (pol[p][row] * v[ch]).sum(1) if q == p else v[ch].sum(1)
                    b[i] = b[ch].max(1).values if q == p else b[ch].sum(1)
                self.up_chance(deal, v, p, 0)
                self.up_chance(deal, b, p, 0)
            root.append((v[0].cpu().numpy(), b[0].cpu().numpy()))
            ev.append(float(v[0] @ self.range[p]))
            br.append(float(b[0] @ self.range[p]))
        mass = float(self.range[0] @ self.C @ self.range[1])
        m = mass if mass > 0 else 1.0
        res = np.array([[br[0] / m, br[1] / m, ev[0] / m, ev[1] / m, mass,
                         0.5 * (br[0] + br[1]) / m / float(self.nd["pot_size"][0])]])
        return res, root[0][0], root[1][0], root[0][1], root[1][1]


def _exact_heads_up(case, seed):
    g = _spot(case, seed, 5 if case["kind"] == "river_spot" else 4)
    if case["kind"] == "turn":
        s = _HeadsUp(g, 0)
        return s.values(s.solve(case["iters"], case["algo"], True, 2.0)[1])
    s = _HeadsUp(g, case["semantics"])
    R, S, cfv = s.solve(case["iters"], case["algo"], case["alternate"], case["avg_power"])
    num = lambda t: t.cpu().numpy()
    return {"R0": num(R[0]), "R1": num(R[1]), "S0": num(S[0]), "S1": num(S[1]), "cfv0": num(cfv[0]),
            "cfv1": num(cfv[1]), "results": s.values(S)[0]}


def _exact_multiway(case, seed):
    g = _multiway_sub(case, seed)
    nd, d, sem, algo = g["nodes"], _dev(), case["semantics"], case["algo"]
    n, H = len(nd), len(g["combos"])
    bub = np.asarray(np.asarray(g["bubble"]).reshape(16).astype(np.float32), np.float64).reshape(4, 4)
    rank = _board_rank(g["board"], g["combos"], _tables())
    own, opp = rank[None, :], rank[:, None]                       # matrices are [opponent hand, own hand]
    if sem == 0:
        C = _disjoint(g["combos"], g["combos"])
        low, tie = (opp < own).double() * C, (opp == own).double() * C
    else:                                                         # rank positions, ties in combo order
        pos = torch.empty(H, dtype=torch.int64, device=d)
        pos[torch.sort(rank, stable=True).indices] = torch.arange(H, device=d)
        C = torch.ones((H, H), dtype=torch.float64, device=d)
        low, tie = (pos[:, None] < pos[None, :]).double(), torch.zeros((H, H), dtype=torch.float64, device=d)
    depth = np.zeros(n, np.int64)
    for i in np.nonzero(nd["type"] == 0)[0]:
        depth[np.arange(nd["num_actions"][i]) + nd["children_offset"][i]] = depth[i] + 1
    levels = [[(p, A, _ints(i), _ints(nd["children_offset"][i])[:, None] + torch.arange(A, device=d),
                _ints(nd["infoset_offset"][i])[:, None] + torch.arange(A, device=d))
               for (p, A), i in _groups((depth == k) & (nd["type"] == 0), nd["player"], nd["num_actions"])]
              for k in range(int(depth.max()) + 1)]
    terms = [(fold, mask, _ints(i), torch.as_tensor(nd["pot_size"][i].astype(np.float64), device=d)[:, None],
              torch.as_tensor(nd["committed"][i].astype(np.float64), device=d))
             for (fold, mask), i in _groups(nd["type"] != 0, nd["type"], nd["active_mask"])]
    z = lambda m: torch.zeros((m, H), dtype=torch.float64, device=d)
    rng = [torch.as_tensor(np.asarray(r, np.float64), device=d) for r in g["ranges"]]
    R, S = [z(r) for r in g["rows"]], [z(r) for r in g["rows"]]
    reach, cfv = [z(n) for _ in range(4)], [z(n) for _ in range(4)]

    def policy(X, floor):
        out = [torch.zeros_like(x) for x in X]
        for lev in levels:
            for p, A, _, _, row in lev:
                pos = X[p][row].clamp(min=0.0)
                s = pos.sum(1, keepdim=True)
                out[p][row] = torch.where(s > floor, pos / torch.where(s > floor, s, torch.ones_like(s)),
                                          torch.full_like(pos, 1.0 / A))
        return out

    def sweep(pol):
        for p in range(4):
            reach[p][0] = rng[p]
        for lev in levels:
            for p, A, i, ch, row in lev:
                for q in range(4):
                    reach[q][ch] = reach[q][i][:, None] * (pol[p][row] if q == p else torch.ones_like(pol[p][row]))
        for fold, mask, i, pot, com in terms:
            W = [reach[o][i] @ C for o in range(4)]
            if fold != 1:
                L, E = [reach[o][i] @ low for o in range(4)], [reach[o][i] @ tie for o in range(4)]
            for p in range(4):
                opps = [o for o in range(4) if o != p]
                c = com[:, p:p + 1]
                if fold == 1 or not mask >> p & 1:
                    win = (mask & -mask).bit_length() - 1
                    pay = pot - c if fold == 1 and p == win else -bub[p, win if fold == 1 else p] * c
                    cfv[p][i] = pay * W[opps[0]] * W[opps[1]] * W[opps[2]]
                    continue
                act, out = [o for o in opps if mask >> o & 1], 1.0
                for o in opps:
                    out = out if mask >> o & 1 else out * W[o]
                share, allw, le = 0.0, 1.0, 1.0
                for o in act:
                    allw, le = allw * W[o], le * (L[o] + E[o])
                for t in range(1 << len(act)):
                    pr = 1.0
                    for k, o in enumerate(act):
                        pr = pr * (E[o] if t >> k & 1 else L[o])
                    share = share + pr * (pot / (1 + bin(t).count("1")) - c)
                cfv[p][i] = (share - bub[p, p] * c * (allw - le)) * out

    def backup(pol, t):
        w = float(t)
        dpos, dneg = ((t - 1.0) ** e / ((t - 1.0) ** e + 1.0) for e in (1.5, 0.0))
        dstr = ((t - 1.0) / t) ** 2.0
        for lev in reversed(levels):
            for p, A, i, ch, row in lev:
                for q in range(4):
                    if q != p:
                        cfv[q][i] = cfv[q][ch].sum(1)
                val = (pol[p][row] * cfv[p][ch]).sum(1)
                cfv[p][i] = val
                if t == 0:
                    continue
                inst, r, add = cfv[p][ch] - val[:, None], R[p][row], reach[p][i][:, None] * pol[p][row]
                R[p][row] = r * torch.where(r > 0, dpos, dneg) + inst if algo else (r + inst).clamp(min=0)
                S[p][row] = S[p][row] * dstr + add if algo else S[p][row] + w * add

    for t in range(1, case["iters"] + 1):
        pol = policy(R, 1e-7)
        sweep(pol)
        backup(pol, t)
    root = np.stack([cfv[p][0].cpu().numpy() for p in range(4)])
    pol = policy(S, 0.0)
    sweep(pol)
    for lev in reversed(levels):
        for p, A, i, ch, row in lev:
            for q in range(4):
                cfv[q][i] = cfv[q][ch].sum(1) if q != p else (pol[p][row] * cfv[p][ch]).sum(1)
    values = np.array([[float(rng[p] @ cfv[p][0]) for p in range(4)]])
    return {"R": [x.cpu().numpy() for x in R], "S": [x.cpu().numpy() for x in S], "cfv": root, "values": values}


def _exact_diff(case, seed):
    subs, sel, packed, r0, r1 = _diff_inputs(case, seed)
    nd, tabs, n = subs[0]["nodes"], _tables(), case["n"]
    H = sel.shape[1]
    rows0 = int(subs[0]["rows"][0])
    shows = [i for i in range(len(nd)) if nd["type"][i] == 2]
    folds = [i for i in range(len(nd)) if nd["type"][i] == 1]
    outs = [[], [], [], []]
    for b0 in range(0, n, 128):
        b1 = min(n, b0 + 128)
        share = torch.empty((b1 - b0, H, H), dtype=torch.float64, device=_dev())
        C = torch.empty_like(share)
        for k in range(b0, b1):
            s = _board_rank(subs[k]["board"], subs[k]["combos0"], tabs)
            C[k - b0] = _disjoint(subs[k]["combos0"], subs[k]["combos1"])
            share[k - b0] = ((s[:, None] > s[None, :]).double() + 0.5 * (s[:, None] == s[None, :]).double()) * C[k - b0]
        lg = packed[b0:b1].double().requires_grad_()
        full = [r[b0:b1].double().requires_grad_() for r in (r0, r1)]
        reach = [[None] * len(nd), [None] * len(nd)]
        for p in (0, 1):
            reach[p][0] = torch.gather(full[p], 1, sel[b0:b1])
        for i in range(len(nd)):
            if nd["type"][i] != 0:
                continue
            p, A, f = int(nd["player"][i]), int(nd["num_actions"][i]), int(nd["children_offset"][i])
            row = int(nd["infoset_offset"][i]) + (rows0 if p else 0)
            pol = torch.softmax(lg[:, row:row + A, :H], 1)
            for a in range(A):
                reach[p][f + a] = reach[p][i] * pol[:, a]
                reach[1 - p][f + a] = reach[1 - p][i]
        at = lambda p, idx: torch.stack([reach[p][i] for i in idx], 1)
        f64 = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=_dev())[None, :, None]
        a0, a1 = at(0, shows), at(1, shows)
        ev = (a0 * (f64(nd["pot_size"][shows]) * torch.bmm(a1, share.transpose(1, 2)) -
                    f64(nd["committed"][shows][:, 0]) * torch.bmm(a1, C))).sum((1, 2))
        pay = np.where(nd["active_mask"][folds] == 1, nd["pot_size"][folds].astype(np.float64), 0.0) \
            - nd["committed"][folds][:, 0]
        ev = ev + (at(0, folds) * f64(pay) * torch.bmm(at(1, folds), C)).sum((1, 2))
        ev.sum().backward()
        for o, v in zip(outs, (ev.detach(), lg.grad.reshape(-1), full[0].grad, full[1].grad)):
            o.append(v)
    return tuple(torch.cat(o) for o in outs)


def _leaf_weights(seed):
    """The network's He initialisation from its seed (splitmix64, Box-Muller), as float32 matrices [out, in]."""
    shapes, live = [(1024, 2752), (1024, 1024), (1024, 1024), (2688, 1024)], [(1024, 2706)] + [(1024, 1024)] * 2 + [(2652, 1024)]
    mask, k0 = (1 << 64) - 1, 0
    st = (seed * 0x9E3779B97F4A7C15 + 0x632BE59BD9B4E019) & mask
    out = []
    with np.errstate(over="ignore"):
        for shape, (o, i) in zip(shapes, live):
            z = np.uint64(st) + np.arange(k0 + 1, k0 + 2 * o * i + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
            k0 += 2 * o * i
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            z ^= z >> np.uint64(31)
            u = ((z >> np.uint64(11)).astype(np.float64) + 0.5) / 9007199254740992.0
            w = np.zeros(shape, np.float32)
            w[:o, :i] = (math.sqrt(2.0 / i) * np.sqrt(-2.0 * np.log(u[0::2])) * np.cos(6.283185307179586 * u[1::2])
                         ).astype(np.float32).reshape(o, i)
            out.append(torch.as_tensor(w, device=_dev()).double())
    return out


def _leaf_forward(W, b, x):
    acts = [torch.nn.functional.pad(x.double(), (0, 2752 - ln.IN))]
    for layer in range(3):
        acts.append(torch.relu(acts[-1] @ W[layer].T + b[layer]))
    return acts, acts[-1] @ W[3].T + b[3]


def _exact_leaf_train(case, seed):
    W = _leaf_weights(seed)
    b = [torch.zeros(w.shape[0], dtype=torch.float64, device=w.device) for w in W]
    x, t, w = _leaf_train_inputs(case, seed)
    par = W + b
    m1, m2 = [torch.zeros_like(p) for p in par], [torch.zeros_like(p) for p in par]
    grads = None
    for k in range(case["steps"]):
        sl = slice(k * case["batch"], (k + 1) * case["batch"])
        acts, y = _leaf_forward(W, b, x[sl])
        d = torch.nn.functional.pad(2.0 * (y[:, :ln.OUT] - t[sl]) / (case["batch"] * ln.OUT) *
                                    (1.0 if w is None else w[sl].double()), (0, 2688 - ln.OUT))
        gw, gb = [None] * 4, [None] * 4
        for layer in (3, 2, 1, 0):
            gw[layer], gb[layer] = d.T @ acts[layer], d.sum(0)
            if layer:
                d = (d @ W[layer]) * (acts[layer] > 0)
        grads = gw + gb
        for p, g, a, v in zip(par, grads, m1, m2):
            a.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).addcmul_(g, g, value=0.001)
            p -= 1e-4 * (a / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    num = lambda v: v.cpu().numpy()
    return [{"w": num(W[i]), "b": num(b[i]), "gw": num(grads[i]), "gb": num(grads[4 + i])} for i in range(4)]


def _combo_class(c1, c2):
    hi, lo = max(c1 // 4, c2 // 4), min(c1 // 4, c2 // 4)
    if hi == lo:
        return 12 - hi
    return (13 if c1 % 4 == c2 % 4 else 91) + sum(r for r in range(12, hi, -1)) + hi - 1 - lo


def _class_cards(cls, mode):
    if cls < 13:
        return (12 - cls) * 4, (12 - cls) * 4 + 1
    base, r1 = (13 if cls < 91 else 91), 12
    off = 0 if cls < 91 else 1
    if mode == 0:                                   # the last class of a rank group runs into the next group
        while r1 > 0 and base + r1 - 1 <= cls:
            base, r1 = base + r1, r1 - 1
        return (4, off) if r1 == 0 else (r1 * 4, (r1 - 1 - (cls - base)) * 4 + off)
    while cls - base >= r1:
        base, r1 = base + r1, r1 - 1
    return r1 * 4, (r1 - 1 - (cls - base)) * 4 + off


def _exact_allin(mode, tabs):
    """3,000 sampled boards per class pair; with replacement in mode 0, without in mode 1."""
    d = _dev()
    pairs = []
    for h in range(169):
        for v in range(169):
            h1, h2 = _class_cards(h, mode)
            v1, v2 = _class_cards(v, mode)
            if mode == 0:
                if v1 in (h1, h2):
                    v1, clash = v1 // 4 * 4 + 2, True
                else:
                    clash = False
                if v2 in (h1, h2):
                    v2 = v2 // 4 * 4 + 3
            elif h != v:
                hi, lo = max(v1, v2) // 4, min(v1, v2) // 4
                v1, v2 = next((hi * 4 + a, lo * 4 + b) for a in range(4) for b in range(4)
                              if ((b > a) if v < 13 else (a == b) if v < 91 else (a != b))
                              and not {hi * 4 + a, lo * 4 + b} & {h1, h2})
            pairs.append((h1, h2, v1, v2))
    decks = np.zeros((len(pairs), 52), np.int64)
    size = np.zeros(len(pairs), np.int64)
    for i, p in enumerate(pairs):
        c = [x for x in range(52) if x not in p]
        decks[i, :len(c)], size[i] = c, len(c)
    deck, size, cards = _ints(decks), _ints(size), _ints(pairs)
    ids = torch.arange(len(pairs), device=d)
    rng = (ids * 2654435761 + 0x9E3779B9) & 0xFFFFFFFF
    win, tie = torch.zeros(len(pairs), device=d).double(), torch.zeros(len(pairs), device=d).double()
    for s0 in range(0, 3000, 50):
        boards = torch.empty((50, 5, len(pairs)), dtype=torch.int64, device=d)
        for s in range(50):
            for k in range(5):
                rng = (rng * 1664525 + 1013904223) & 0xFFFFFFFF
                pick = (k + (rng >> 16) % (size - k))[:, None]
                c = deck.gather(1, pick)
                if mode:
                    deck.scatter_(1, pick, deck[:, k:k + 1])
                    deck[:, k:k + 1] = c
                boards[s, k] = c[:, 0]
        b = [boards[:, k] for k in range(5)]
        a, v = (_rank([cards[None, :, j], cards[None, :, j + 1]] + b, tabs) for j in (0, 2))
        win += (a > v).double().sum(0)
        tie += (a == v).double().sum(0)
    out = ((win + 0.5 * tie) / 3000.0).reshape(169, 169)
    out.fill_diagonal_(0.5)
    return out


def _exact_flop_class(flop, mode, tabs):
    d = _dev()
    combos = _PAIRS[:1176] if mode == 0 else _PAIRS
    n = len(combos)
    deck = [c for c in range(52) if c not in flop]
    runs = [(deck[i], deck[j]) for i in range(49) for j in range(i + 1, 49)]
    slot = {r: k for k, r in enumerate(runs)}
    rt, cc = _ints(runs), _ints(combos)
    key = _rank([_ints(int(c)) for c in flop] + [rt[:, None, 0], rt[:, None, 1], cc[None, :, 0], cc[None, :, 1]], tabs)
    hits = (rt[:, None, :, None] == cc[None, :, None, :]).any(-1).any(-1)          # runout touches the combo
    key = torch.where(hits, torch.full_like(key, -1), key)
    onflop = np.isin(combos, flop).any(axis=1)
    E = torch.zeros((n, n), dtype=torch.float64, device=d)                         # [hero, villain]
    lists = []
    for h in np.nonzero(~onflop)[0]:
        own = [c for c in deck if c not in combos[h]]
        lists.append([slot[own[a], own[b]] for a in range(0, 47, 2) for b in range(a + 1, 47, 3)])
    heroes = np.nonzero(~onflop)[0]
    free = _disjoint(np.arange(n), np.arange(n)) * torch.as_tensor(~onflop, device=d).double()[None, :]
    for k in range(0, len(heroes), 32):
        hs, ls = _ints(heroes[k:k + 32]), _ints(lists[k:k + 32])
        hk, vk = key[ls, hs[:, None]][:, :, None], key[ls]
        tot = (vk >= 0).double().sum(1)
        win = ((hk > vk) & (vk >= 0)).double().sum(1)
        tie = ((hk == vk) & (vk >= 0)).double().sum(1)
        eq = (win + tie * (0.25 if mode == 0 else 0.5)) / tot.clamp(min=1.0)
        E[hs] = eq * free[hs]
    cls = np.array([_combo_class(int(a), int(b)) for a, b in combos])
    M = torch.zeros((169, n), dtype=torch.float64, device=d)
    M[_ints(cls), torch.arange(n, device=d)] = 1.0
    tot, cnt = M @ E @ M.T, M @ (E > 0).double() @ M.T
    return torch.where(cnt > 0, tot / cnt.clamp(min=1.0), torch.full_like(tot, 0.5)).T


def _exact_dcfr(weights, mats, allin, iters, stack=20.0, bf=1.35, dead=2.5):
    d = _dev()
    w = torch.as_tensor(np.asarray(weights, np.float64), device=d)
    bf = float(np.float32(bf))
    acts = (3, 3, 2, 2)
    root = torch.as_tensor(np.where(np.arange(169) < 13, 6.0, np.where(np.arange(169) < 91, 4.0, 12.0)) / 1326.0, device=d)
    G = [torch.full((a, 169), 1.0 / a, dtype=torch.float64, device=d) for a in acts]
    R, S = [torch.zeros_like(g) for g in G], [torch.zeros_like(g) for g in G]
    jam_net = stack + dead
    jam = lambda eq: eq * jam_net - (1.0 - eq) * bf * stack
    div = lambda a, m: a / m if m > 1e-7 else a
    net = lambda x: torch.where(x >= 2.1, x - 2.1, -(2.1 - x) * bf)
    for t in range(1, iters + 1):
        wp, ws = t ** 1.5 / (t ** 1.5 + 1.0), float(t) * t
        rbc, rbb = root * G[0][1], root * G[1][1]
        e0 = div(torch.einsum("o,foc->fc", rbb, mats), rbb.sum())
        e1 = div(torch.einsum("o,fco->fc", rbc, 1.0 - mats), rbc.sum())
        evb = (w[:, None] * net(e0 * 1.06 * (dead + 3.1))).sum(0) / w.sum()
        evbb = (w[:, None] * net(e1 * 0.94 * (dead + 3.1))).sum(0) / w.sum()
        br, bd, b3, bj = G
        m3 = root * bd[2]
        c3 = torch.stack([torch.full_like(root, -2.1 * bf), jam(div(allin @ m3, m3.sum()))])
        v3 = (b3 * c3).sum(0)
        ro = root * br[1]
        f3, k3 = (ro * b3[0]).sum(), ro * b3[1]
        evsh = jam(div((1.0 - allin).T @ k3, k3.sum()))
        cd = torch.stack([torch.full_like(root, -bf), evbb, (f3 * (dead + 2.1) + k3.sum() * evsh) / (f3 + k3.sum() + 1e-9)])
        mj = root * br[2]
        cj = torch.stack([torch.full_like(root, -bf), jam(div((1.0 - allin).T @ mj, mj.sum()))])
        f, c, j = (root * bd[0]).sum(), (root * bd[1]).sum(), (root * bd[2]).sum()
        fj, kj = (root * bj[0]).sum(), root * bj[1]
        evj = jam(div(allin @ kj, kj.sum()))
        cr = torch.stack([torch.zeros_like(root), (f * dead + c * evb + j * v3) / (f + c + j + 1e-9),
                          (fj * dead + kj.sum() * evj) / (fj + kj.sum() + 1e-9)])
        for k, C in enumerate((cr, cd, c3, cj)):
            v = (G[k] * C).sum(0)
            S[k] = S[k] + ws * root * G[k]
            R[k] = wp * (R[k] + C - v).clamp(min=0.0)
            pos = R[k].sum(0, keepdim=True)
            G[k] = torch.where(pos > 1e-7, R[k] / pos.clamp(min=1e-300), torch.full_like(R[k], 1.0 / acts[k]))
    pad = lambda x: torch.nn.functional.pad(torch.cat(x), (0, 23))
    out = pad(G)
    for k, a in enumerate(acts):                      # the padding columns keep the uniform start
        out[sum(acts[:k]):sum(acts[:k]) + a, 169:] = 1.0 / a
    return pad(S), out


def _exact_dump(case, seed):
    """The dump's definition: a subsample of runouts, every fourth villain, uniform reach, summed per class."""
    d, tabs = _dev(), _tables()
    out = []
    runs = [(a, b) for a in range(0, 47, 2) for b in range(a + 1, 47, 3)]
    for flop in _flops(case["n"], seed)[0]:
        deck = np.array([c for c in range(52) if c not in flop])
        hands = np.array([(a, b) for i, a in enumerate(deck) for b in deck[i + 1:]])
        rt, cc = _ints(deck[np.array(runs)]), _ints(hands)
        key = _rank([_ints(int(c)) for c in flop] + [rt[:, None, 0], rt[:, None, 1], cc[None, :, 0], cc[None, :, 1]], tabs)
        use = ~(rt[:, None, :, None] == cc[None, :, None, :]).any(-1).any(-1)
        key = torch.where(use, key, torch.full_like(key, -1)).to(torch.int32)
        hk, vk = key[:, :, None], key[:, None, ::4]
        both = (hk >= 0) & (vk >= 0)
        n = both.sum(0).double()
        eq = (((hk > vk) & both).sum(0) + 0.5 * ((hk == vk) & both).sum(0)) / n.clamp(min=1.0)
        ok = (cc[:, None, :, None] != cc[None, ::4, None, :]).all(-1).all(-1) & (n > 0)
        ev = torch.where(ok, 2.0 * eq - 1.0, torch.zeros_like(eq)).sum(1) / 1176.0
        cls = _ints([_combo_class(int(a), int(b)) for a, b in hands])
        tot = torch.zeros(169, dtype=torch.float64, device=d).index_add_(0, cls, ev)
        out.append(torch.stack([torch.stack([tot, -tot]) * (1.0 + 0.1 * s) for s in range(4)]))
    return torch.stack(out)


def exact(case, seed):
    k = case["kind"]
    if k in ("eval7", "counts"):          # whole numbers
        return None
    if k == "river_batch":                # thousands of trees: minutes in 64 bits
        return None
    if k == "dump":
        return _exact_dump(case, seed)
    if k in ("river_spot", "turn"):
        return _exact_heads_up(case, seed)
    if k == "diff_ev":
        return _exact_diff(case, seed)
    if k == "multiway":
        return _exact_multiway(case, seed)
    if k == "leaf_rows":
        W = _leaf_weights(seed)
        b = [torch.zeros(w.shape[0], dtype=torch.float64, device=w.device) for w in W]
        return _leaf_forward(W, b, _leaf_features(case["rows"], seed)[0])[1][:, :ln.OUT]
    if k == "leaf_train":
        return _exact_leaf_train(case, seed)
    flops, weights = _flops(case["flops"], seed)
    tabs = _tables()
    allin = _exact_allin(case["mode"], tabs)
    mats = torch.stack([_exact_flop_class([int(c) for c in f], case["mode"], tabs) for f in flops])
    sums, sigma = _exact_dcfr(weights, mats, allin, case["iters"])
    return allin, mats, sums, sigma

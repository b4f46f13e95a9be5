"""The work that a program has this solver do, as cases that can be timed.

Each case is one call of a public entry point over inputs drawn from a seed:

  solve    a single-street subgame from host buffers to host outputs
           (StreetSolverGPU.solve): the call a real-time player makes once per
           street, from a narrowed heads-up river to a full-range turn of three
           or four players with continuation leaves
  batch    many subgames of mixed streets, sizes and player counts solved
           together to an exploitability target (ss_batch_solve)
  exploit  the FP64 exploitability of a given profile (ss_exploitability_gpu)
  leaves   the continuation values that a depth-limited turn or flop needs
           before its solve (leaf_values.compute_*)
  flop     the flop-through-river solver (fs_solve_gpu)

Ranges, boards and leaf values follow the benchmark's distributions: boards are
random, weights U(0, 1) with a share of them zero, leaf values N(0, 0.3 pot).
exact() restates the algorithm in 64 bits with plain torch and numpy.
"""
import ctypes
import itertools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "poker-solver_b200"))
import flop_solve as fsm  # noqa: E402
import leaf_values as lvm  # noqa: E402
import street_solver_gpu as ssg  # noqa: E402
import workloads as wl  # noqa: E402


def _solve(name, players, street, bets, raises, iterations, hands=0, zero=0.0, pot=100, stack=400):
    c = {"kind": "solve", "players": players, "board": {"flop": 3, "turn": 4, "river": 5}[street], "hands": hands,
         "zero": zero, "bets": bets, "raises": raises, "pot": pot, "stack": stack, "iterations": iterations}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a heads-up river after two streets of narrowing: the smallest solve,
        # with the class's default bet sizes, raise cap and iterations
        _solve("river_hu_narrow", 2, "river", "0.33,0.75,1.5", 3, 200, hands=90),
        # the heads-up river configuration: every combo, 1000 iterations
        _solve("river_hu_full", 2, "river", "0.5,1.0", 2, 1000),
        # a heads-up turn with continuation leaves, every combo
        _solve("turn_hu_full", 2, "turn", "0.33,0.75,1.5", 3, 200, pot=150, stack=500),
        # a three-player river, every combo (three-way showdowns)
        _solve("river3_full", 3, "river", "0.5,1.0", 2, 200, pot=300, stack=1000),
        # the headline turn: three players, 21,436 nodes, every combo, 30% of the weights zero
        _solve("turn3_full", 3, "turn", "0.33,0.75,1.5", 3, 200, zero=0.3, pot=150, stack=500),
        # a four-player river after narrowing (four-way showdowns over sparse ranges)
        _solve("river4_narrow", 4, "river", "0.5,1.0", 2, 20, hands=101, zero=0.35),
        # a four-player turn at full ranges: terminals with three counted opponents
        _solve("turn4_full", 4, "turn", "1.0", 1, 4, zero=0.3, pot=150, stack=500),
        # one batch of a solver that serves many tables: all streets, 2 to 6 players
        {"name": "batch_mixed", "kind": "batch", "requests": 16, "iterations": 200, "target": 0.5},
        # how far a given profile of the three-player turn is from equilibrium
        {"name": "exploit_turn3", "kind": "exploit", "players": 3, "board": 4, "hands": 0, "zero": 0.3,
         "bets": "0.33,0.75,1.5", "raises": 2, "pot": 150, "stack": 500},
        # continuation values of a narrow heads-up turn (a small call) ...
        {"name": "leaves_turn_hu", "kind": "leaves", "players": 2, "board": 4, "hands": 40, "zero": 0.0,
         "bets": "0.5,1.0", "raises": 2, "pot": 100, "stack": 400},
        # ... and of the headline turn
        {"name": "leaves_turn3", "kind": "leaves", "players": 3, "board": 4, "hands": 0, "zero": 0.3,
         "bets": "0.33,0.75,1.5", "raises": 3, "pot": 150, "stack": 500},
        # flop through river, 574,638 nodes, the ABI's largest ranges
        {"name": "flop_river", "kind": "flop", "hands": 200, "bets": "0.75", "pot": 100, "stack": 10000,
         "iterations": 50},
    ]


# bet sets and raise caps of the request mix; the larger ones only where the
# tree stays within the headline turn's size
_BETS = ["1.0", "0.75", "0.5", "0.5,1.0", "0.33,0.75", "0.33,0.75,1.5", "0.25,0.5,1.0,2.0"]


def _between(rng, lo, hi):
    """A whole number, uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choices(["hu", "three", "four", "exploit", "leaves", "flop", "batch"], [6, 4, 2, 2, 2, 1, 1])[0]
    pot = 50 * rng.randint(1, 8)
    stack = pot * rng.randint(2, 8)
    zero = round(rng.uniform(0.0, 0.7), 3)
    bets = rng.choice(_BETS)
    if what == "hu":
        street = rng.choice(["river", "river", "turn", "flop"])
        return _solve("", 2, street, bets, rng.randint(1, 3), _between(rng, 10, 300),
                      hands=_between(rng, 13, 1081), zero=zero, pot=pot, stack=stack)
    if what == "three":
        street = rng.choice(["river", "turn"])
        raises = rng.randint(1, 3) if street == "river" else rng.randint(1, 2)
        return _solve("", 3, street, bets if street == "river" else rng.choice(_BETS[:5]), raises,
                      _between(rng, 4, 100), hands=_between(rng, 20, 1081), zero=zero, pot=pot, stack=stack)
    if what == "four":
        if rng.random() < 0.5:
            return _solve("", 4, "river", rng.choice(_BETS[:4]), 1, rng.randint(2, 6),
                          hands=_between(rng, 24, 1081), zero=zero, pot=pot, stack=stack)
        return _solve("", 4, "turn", rng.choice(_BETS[:3]), 1, rng.randint(2, 3),
                      hands=_between(rng, 24, 1081), zero=zero, pot=pot, stack=stack)
    if what == "exploit":
        return {"kind": "exploit", "players": rng.randint(2, 3), "board": rng.choice([4, 5]),
                "hands": _between(rng, 20, 1081), "zero": zero, "bets": rng.choice(_BETS[:5]),
                "raises": rng.randint(1, 2), "pot": pot, "stack": stack}
    if what == "leaves":
        players = rng.randint(2, 3)
        return {"kind": "leaves", "players": players, "board": rng.choice([3, 4]), "hands": _between(rng, 12, 1128),
                "zero": 0.0, "bets": rng.choice(_BETS[:5]), "raises": rng.randint(1, 2), "pot": pot, "stack": stack}
    if what == "flop":
        return {"kind": "flop", "hands": _between(rng, 20, 199), "bets": rng.choice(_BETS[:3]), "pot": pot,
                "stack": stack * 10, "iterations": _between(rng, 4, 40)}
    return {"kind": "batch", "requests": rng.randint(4, 12), "iterations": 25 * rng.randint(2, 6),
            "target": rng.choice([0.25, 0.5, 1.0])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _bets(case):
    return [float(x) for x in case["bets"].split(",")]


def _board_and_ranges(case, seed):
    """Random board; per player `hands` distinct combos of the rest of the deck
    (0: all of them) in ascending order, weights U(0, 1), a share `zero` of them 0."""
    rng = np.random.default_rng(seed)
    board = [int(c) for c in rng.permutation(52)[:case["board"]]]
    combos = np.array([(a, b) for a in range(52) for b in range(a + 1, 52) if a not in board and b not in board],
                      np.int32)
    hands, weights = [], []
    for _ in range(case["players"]):
        n = case["hands"] or len(combos)
        at = np.arange(len(combos)) if n >= len(combos) else np.sort(rng.choice(len(combos), n, replace=False))
        w = rng.uniform(0.0, 1.0, len(at))
        w[rng.random(len(at)) < case["zero"]] = 0.0
        hands.append(combos[at])
        weights.append(w.astype(np.float32))
    return board, hands, weights


def _leaf_values(case, seed, num_leaves, max_h):
    if num_leaves == 0:
        return None
    rng = np.random.default_rng(seed + 1000)
    lv = rng.standard_normal((num_leaves, case["players"], max_h), dtype=np.float32)
    lv *= np.float32(0.3 * case["pot"])
    return lv


def _subgame(case, seed, wide=False):
    """The subgame through the C-ABI driver: tree built, ranges and leaf values filled."""
    board, hands, weights = _board_and_ranges(case, seed)
    sg = wl.AbiSubgame(dict(board=board, pot=case["pot"], stack=case["stack"], bet_sizes=_bets(case),
                            max_raises=case["raises"], num_players=case["players"], hands=hands, weights=weights),
                       max_hands=ssg.SS_MAX_HANDS_WIDE if wide else None)
    sg.set_leaf_values(_leaf_values(case, seed, sg.num_leaves, max(len(h) for h in hands)))
    return sg


# the batch's requests, in turn: street, players, bets, raises, hands per player
_REQUESTS = [("river", 2, "0.5,1.0", 2, 0), ("turn", 2, "0.33,0.75", 2, 0), ("river", 3, "0.75", 2, 0),
             ("flop", 2, "0.5,1.0", 1, 0), ("river", 4, "0.5", 2, 80), ("turn", 3, "0.5", 1, 0),
             ("river", 2, "0.25,0.5,1.0,2.0", 3, 300), ("river", 5, "1.0", 1, 6), ("turn", 2, "1.0", 2, 500),
             ("flop", 3, "1.0", 1, 400), ("river", 6, "1.0", 1, 4), ("river", 3, "0.5,1.0", 1, 200)]


def _request_case(i):
    street, players, bets, raises, hands = _REQUESTS[i % len(_REQUESTS)]
    return _solve("", players, street, bets, raises, 0, hands=hands, zero=0.05 * (i % 13), pot=50 + 25 * (i % 11),
                  stack=4 * (50 + 25 * (i % 11)))


def _profile(na, owner, num_hands, max_h, seed):
    """A random profile in the output layout: per decision node and hand a
    distribution over its actions (na[i] actions, acting player owner[i])."""
    rng = np.random.default_rng(seed + 2000)
    p = rng.random((len(na), ssg.SS_MAX_ACTIONS, max_h), dtype=np.float32)
    for a in range(ssg.SS_MAX_ACTIONS):
        p[na <= a, a] = 0.0
    for q, n in enumerate(num_hands):
        p[owner == q, :, n:] = 0.0
    s = p.sum(axis=1, keepdims=True)
    return p / np.where(s > 0, s, np.float32(1.0))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        board, hands, weights = _board_and_ranges(case, seed)
        ranges = [[(int(a), int(b), float(x)) for (a, b), x in zip(h, w)] for h, w in zip(hands, weights)]
        n = max(len(r) for r in ranges)
        s = ssg.StreetSolverGPU(board, case["pot"] / 100, case["stack"] / 100, player_ranges=ranges,
                                bet_sizes=_bets(case), max_raises=case["raises"],
                                leaf_value_fn=lambda tree, ph, mh, pot: _leaf_values(case, seed, tree.num_leaves, mh),
                                max_hands=ssg.SS_MAX_HANDS if n <= ssg.SS_MAX_HANDS else ssg.SS_MAX_HANDS_WIDE)
        return {"case": case, "solver": s}
    if kind == "batch":
        subs = [_subgame(_request_case(i), 1000 * seed + i, wide=True) for i in range(case["requests"])]
        return {"case": case, "subgames": subs}
    if kind == "exploit":
        sg = _subgame(case, seed)
        nodes = sg.tree_arrays()[0]
        dec = nodes[nodes[:, 0] == ssg.NODE_DECISION]
        avg = _profile(dec[:, 2], dec[:, 1], sg.nh, int(sg.nh.max()), seed)
        return {"case": case, "subgame": sg, "avg": avg}
    if kind == "leaves":
        board, hands, weights = _board_and_ranges(case, seed)
        sg = wl.AbiSubgame(dict(board=board, pot=case["pot"], stack=case["stack"], bet_sizes=_bets(case),
                                max_raises=case["raises"], num_players=case["players"], hands=hands, weights=weights))
        infos = lvm.extract_leaf_info_from_tree(sg.td, case["players"])
        ranges = [[(int(a), int(b), float(x)) for (a, b), x in zip(h, w)] for h, w in zip(hands, weights)]
        return {"case": case, "board": board, "infos": infos, "ranges": ranges,
                "max_hands": max(len(r) for r in ranges)}
    # flop through river
    three = dict(case, board=3, players=2, zero=0.0)
    board, hands, weights = _board_and_ranges(three, seed)
    return {"case": case, "subgame": fsm.FlopSubgame(ssg.load_library(), board, case["pot"], case["stack"],
                                                     _bets(case), hands, weights)}


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------

def _view(owner, ptr, shape):
    """The solver's own output buffer as an array that keeps the solver alive."""
    buf = (ctypes.c_float * int(np.prod(shape))).from_address(ctypes.addressof(ptr.contents))
    buf.owner = owner
    return np.frombuffer(buf, np.float32).reshape(shape)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        s = state["solver"]
        s.solve(case["iterations"])
        o = s._output
        nh = len(s.player_hands[o.root_player])
        return {"avg": _view(s, o.avg_strategies, (o.num_avg_nodes, ssg.SS_MAX_ACTIONS, o.max_hands)),
                "root": _view(s, o.root_strategy, (o.root_num_actions, nh)),
                "ev": _view(s, o.root_ev, (o.max_hands,))}
    if kind == "batch":
        rc, res = wl.batch_solve(state["subgames"], case["iterations"], target=case["target"])
        if rc != 0:
            raise RuntimeError(f"ss_batch_solve failed ({rc}): {ssg.last_error(state['subgames'][0].lib)}")
        return [{"avg": r["avg_strategies"], "root": r["root_strategy"], "ev": r["root_ev"]} for r in res]
    if kind == "exploit":
        sg = state["subgame"]
        pct, nash, z = ctypes.c_double(), ctypes.c_double(), ctypes.c_double()
        br, cur = (ctypes.c_double * ssg.SS_MAX_PLAYERS)(), (ctypes.c_double * ssg.SS_MAX_PLAYERS)()
        rc = sg.lib.ss_exploitability_gpu(ctypes.byref(sg.td), state["avg"].ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                                          ctypes.byref(pct), ctypes.byref(nash), br, cur, ctypes.byref(z))
        if rc != 0:
            raise RuntimeError(f"ss_exploitability_gpu failed ({rc}): {ssg.last_error(sg.lib)}")
        n = case["players"]
        return {"pct": pct.value, "nash": nash.value, "br": np.array(br[:n]), "cur": np.array(cur[:n]), "mass": z.value}
    if kind == "leaves":
        f = lvm.compute_turn_leaf_values if case["board"] == 4 else lvm.compute_flop_leaf_equity
        return f(state["board"], state["infos"], state["max_hands"], case["pot"], player_hands=state["ranges"])
    return state["subgame"].solve(case["iterations"])["root_strategy"]


# ---------------------------------------------------------------------------
# the betting tree, from its rules (for work() and exact())
# ---------------------------------------------------------------------------

class _Tree:
    """Nodes in the solver's numbering: a decision before its subtrees; then
    every leaf's chain of 4-way continuation choices, one level per live player."""

    def __init__(self, case):
        self.n = case["players"]
        self.river = case["board"] == 5
        self.sizes = [np.float32(b) for b in _bets(case)]
        self.raises = case["raises"]
        self.kind, self.player, self.kids, self.pot, self.bets, self.live, self.leaf = [], [], [], [], [], [], []
        one = (1,) * self.n
        self._grow(0, case["pot"], case["stack"], (0,) * self.n, (0,) * self.n, one, 0)
        if not self.river:
            self._expand()

    def _make(self, kind, pot, bets, live):
        for col, v in ((self.kind, kind), (self.player, -1), (self.kids, []), (self.pot, pot), (self.bets, bets),
                       (self.live, live), (self.leaf, -1)):
            col.append(v)
        return len(self.kind) - 1

    def _grow(self, seat, pot, stack, bets, acted, live, raises):
        n = self.n
        top = max(b for b, v in zip(bets, live) if v)
        if sum(live) <= 1:
            x = self._make("fold", pot, bets, live)
            self.player[x] = live.index(1)
            return x
        if all(not v or (a and b == top) for v, a, b in zip(live, acted, bets)):
            return self._make("showdown" if self.river else "leaf", pot, bets, live)
        while not live[seat]:
            seat = (seat + 1) % n
        x = self._make("decision", pot, bets, live)
        self.player[x] = seat
        call = top - bets[seat]
        nxt = next((seat + k) % n for k in range(1, n + 1) if live[(seat + k) % n])

        def put(t, v):
            return t[:seat] + (v,) + t[seat + 1:]

        kids = []
        if call > 0:
            kids.append(self._grow(nxt, pot, stack, bets, acted, put(live, 0), raises))
        kids.append(self._grow(nxt, pot + call, stack, put(bets, top), put(acted, 1), live, raises))
        if raises < self.raises:
            amounts, allin = [], False
            for f in self.sizes:
                a = int(f * np.float32(pot)) if call == 0 else call + int(f * np.float32(pot + call))
                a = min(a, stack)
                if a <= call or (a >= stack and allin):
                    continue
                allin = allin or a >= stack
                amounts.append(a)
            if not allin and stack > call:
                amounts.append(stack)
            for a in amounts:
                again = tuple(1 if p == seat else 0 if live[p] else acted[p] for p in range(n))
                kids.append(self._grow(nxt, pot + a, stack, put(bets, top + a), again, live, raises + 1))
        self.kids[x] = kids
        return x

    def _expand(self):
        self.chain_heads = []     # (index of the chain's first leaf, pot) of the chains of all players
        leaves = 0
        for x in [i for i, k in enumerate(self.kind) if k == "leaf"]:
            chain = [p for p in range(self.n) if self.live[x][p]]
            layer = [x]
            for step, p in enumerate(chain):
                below = []
                for y in layer:
                    self.kind[y], self.player[y] = "decision", p
                    self.kids[y] = [self._make("leaf", self.pot[x], self.bets[x], self.live[x]) for _ in range(4)]
                    below += self.kids[y]
                layer = below
            if len(chain) == self.n:
                self.chain_heads.append((leaves, self.pot[x]))
            for y in layer:
                self.leaf[y] = leaves
                leaves += 1
        self.num_leaves = leaves


def _counted(tree, x, t):
    """The opponents whose hands count at terminal x for traverser t (None: the value is 0)."""
    if tree.kind[x] == "fold":
        return [o for o in range(tree.n) if o != t]
    if tree.kind[x] == "showdown" and not tree.live[x][t]:
        return None
    return [o for o in range(tree.n) if o != t and tree.live[x][o]]


def _solve_work(case, iterations):
    """Bytes and operations of `iterations` of the solve: inputs and outputs
    once; per iteration and decision edge the regrets and strategy sums read
    and written, the reach written and read; per terminal its opponents' reach
    and leaf values read, its value written and read; a two-card matrix
    product per pair of counted opponents and a few operations per hand."""
    tree = _Tree(case)
    deck = 52 - case["board"]
    H = min(case["hands"] or 10 ** 9, deck * (deck - 1) // 2)
    edges = sum(len(k) for k in tree.kids)
    decisions = sum(1 for k in tree.kids if k)
    byt, flops = iterations * edges * H * 24.0, iterations * edges * H * 12.0
    leaf_bytes = 0.0
    for x in range(len(tree.kind)):
        if tree.kids[x]:
            continue
        for t in range(tree.n):
            opp = _counted(tree, x, t)
            k = len(opp) if opp is not None else 0
            byt += iterations * 4.0 * H * (k + 2 + (tree.kind[x] == "leaf"))
            flops += iterations * (max(0, k - 1) * 2.0 * deck ** 3 + 20.0 * H * k)
        leaf_bytes += 4.0 * H * tree.n if tree.kind[x] == "leaf" else 0.0
    return {"bytes": byt + leaf_bytes + 4.0 * 8 * decisions * H, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "solve":
        return _solve_work(case, case["iterations"])
    if kind == "batch":
        # about half of the iteration cap is run before the target is met
        w = [_solve_work(_request_case(i), case["iterations"] // 2) for i in range(case["requests"])]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if kind == "exploit":
        w = _solve_work(case, 1)
        return {"bytes": 2.0 * w["bytes"], "flops": w["flops"]}
    if kind == "leaves":
        tree = _Tree(case)
        deck = 52 - case["board"]
        H = min(case["hands"] or 10 ** 9, deck * (deck - 1) // 2)
        n = case["players"]
        runouts = 12 ** (5 - case["board"]) if H > 50 else math.prod(range(48, 53 - case["board"]))
        tuples = min(2000, (H + 0.0) ** (n - 1))
        values = len(tree.chain_heads) * 4 ** n * n * H
        return {"bytes": 4.0 * values + 12.0 * n * H, "flops": 4.0 * runouts * n * H * tuples + 6.0 * values}
    # flop through river: the decisions' rows as in a street solve; about a
    # third of the tree's edges are decision edges of each player
    flop_bets = len(_bets(case))
    edges = 287_000.0 * (1 + flop_bets)
    return {"bytes": case["iterations"] * edges * 24.0 * case["hands"], "flops": case["iterations"] * edges * 12.0 * case["hands"]}


# ---------------------------------------------------------------------------
# the same values in 64 bits
# ---------------------------------------------------------------------------

def _strengths(board5, hands):
    """7-card strengths as whole numbers that order hands (0: a card repeats)."""
    cards = np.concatenate([np.broadcast_to(np.array(board5), (len(hands), 5)), hands], axis=1)
    rank, suit = cards // 4, cards % 4
    best = np.zeros(len(hands), np.int64)
    for five in itertools.combinations(range(7), 5):
        r, s = -np.sort(-rank[:, five], axis=1), suit[:, five]
        flush = (s == s[:, :1]).all(axis=1)
        count = (r[:, :, None] == r[:, None, :]).sum(axis=2)
        # ranks by multiplicity, then by rank
        order = np.argsort(-(count * 16 + r), axis=1, kind="stable")
        key = np.take_along_axis(r, order, axis=1)
        c = np.take_along_axis(count, order, axis=1)
        distinct = (c == 1).all(axis=1)
        wheel = distinct & (key == np.array([12, 3, 2, 1, 0])).all(axis=1)
        straight = distinct & (key[:, 0] - key[:, 4] == 4) | wheel
        key = np.where(wheel[:, None], np.array([3, 2, 1, 0, 0]), key)
        cat = np.select([straight & flush, c[:, 0] == 4, (c[:, 0] == 3) & (c[:, 3] == 2), flush, straight, c[:, 0] == 3,
                         (c[:, 0] == 2) & (c[:, 2] == 2), c[:, 0] == 2], [8, 7, 6, 5, 4, 3, 2, 1], 0)
        v = cat
        for i in range(5):
            v = v * 16 + key[:, i]
        best = np.maximum(best, v + 1)
    twice = (np.sort(cards, axis=1)[:, 1:] == np.sort(cards, axis=1)[:, :-1]).any(axis=1)
    return np.where(twice, 0, best)


class _Game:
    """The subgame in FP64 tensors: reach and values per node, terminal values
    by the card-removal closed forms (one and two counted opponents)."""

    def __init__(self, case, seed):
        self.case, self.tree = case, _Tree(case)
        tr = self.tree
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        board, hands, weights = _board_and_ranges(case, seed)
        self.n = tr.n
        self.H = [len(h) for h in hands]
        self.mh = max(self.H)
        N = self.N = len(tr.kind)
        A = ssg.SS_MAX_ACTIONS
        f64 = torch.float64
        self.depth = np.zeros(N, int)
        for x in range(N):
            for y in tr.kids[x]:
                self.depth[y] = self.depth[x] + 1
        self.dec = [x for x in range(N) if tr.kids[x]]
        self.na = np.array([len(tr.kids[x]) for x in self.dec])
        self.owner = np.array([tr.player[x] for x in self.dec])
        kids = np.full((len(self.dec), A), N)
        for i, x in enumerate(self.dec):
            kids[i, :len(tr.kids[x])] = tr.kids[x]
        self.kids = torch.tensor(kids, device=self.dev)
        self.legal = self.kids < N
        dec_depth = self.depth[self.dec]
        self.levels = []       # (depth order) decision indices per (depth, player)
        for d in range(int(dec_depth.max()) + 1):
            self.levels.append([(p, torch.tensor(np.flatnonzero((dec_depth == d) & (self.owner == p)), device=self.dev))
                                for p in range(self.n) if ((dec_depth == d) & (self.owner == p)).any()])
        self.dec_t = torch.tensor(self.dec, device=self.dev)
        self.hand = [torch.tensor(h.astype(np.int64), device=self.dev) for h in hands]
        self.weight = [torch.tensor(w.astype(np.float64), device=self.dev) for w in weights]
        self.reach = [torch.zeros(N + 1, h, dtype=f64, device=self.dev) for h in self.H]
        self.share = [[(self.hand[t][:, None, :, None] == self.hand[o][None, :, None, :]).any(3).any(2)
                       for o in range(self.n)] for t in range(self.n)]
        if tr.river:
            self.str = [torch.tensor(_strengths(board, h), device=self.dev) for h in hands]
        lv = _leaf_values(case, seed, getattr(tr, "num_leaves", 0), self.mh) if not tr.river else None
        self.leaf = None if lv is None else torch.tensor(lv, device=self.dev)
        # per traverser, the terminals by kind and counted opponents
        self.terms = []
        for t in range(self.n):
            groups = {}
            for x in range(N):
                if tr.kids[x]:
                    continue
                opp = _counted(tr, x, t)
                if opp is not None:
                    groups.setdefault((tr.kind[x], tuple(opp)), []).append(x)
            self.terms.append(groups)

    def set_reach(self, p, sigma):
        """Player p's reach of every node; sigma [decisions, 8, hands]."""
        r = self.reach[p]
        r[0] = self.weight[p]
        for level in self.levels:
            for q, at in level:
                up = r[self.dec_t[at]][:, None, :].expand(-1, ssg.SS_MAX_ACTIONS, -1)
                r[self.kids[at]] = up * sigma[at][:, :, :self.H[p]] if q == p else up

    def pairs(self, t, o1, o2, r1, r2, at=None):
        """Mass of disjoint pairs of opponent hands avoiding each of t's hands
        (those at `at`): [rows, hands], 0 exactly where no pair has positive reach."""
        h = self.hand[t] if at is None else self.hand[t][at]
        a, b = h[:, 0], h[:, 1]

        def form(x1, x2):
            M = []
            for o, x in ((o1, x1), (o2, x2)):
                m = torch.zeros(x.shape[0], 52, 52, dtype=torch.float64, device=self.dev)
                c, d = self.hand[o][:, 0], self.hand[o][:, 1]
                m[:, c, d] = x
                m[:, d, c] = x
                M.append(m)
            M1, M2 = M
            u1, u2 = M1.sum(2), M2.sum(2)
            P = torch.bmm(M1, M2)
            w = P.sum(2) + P.sum(1)
            d = torch.diagonal(P, dim1=1, dim2=2)
            F1, F2 = u1.sum(1, keepdim=True) / 2, u2.sum(1, keepdim=True) / 2
            g = u1 * u2 + w - 2 * d
            rest = d.sum(1, keepdim=True) / 2 - (u1 * u2).sum(1, keepdim=True)
            m1, m2 = M1[:, a, b], M2[:, a, b]
            s1, s2 = u1[:, a] + u1[:, b], u2[:, a] + u2[:, b]
            return ((F1 - s1 + m1) * (F2 - s2 + m2) + rest + g[:, a] + g[:, b] - m2 * s1 - m1 * s2 + 3 * m1 * m2 -
                    P[:, a, b] - P[:, b, a])

        out = []
        for i in range(0, r1.shape[0], 2048):
            x, y = r1[i:i + 2048], r2[i:i + 2048]
            out.append(torch.where(form((x > 0).double(), (y > 0).double()) > 0.5, form(x, y), 0.0))
        return torch.cat(out)

    def terminals(self, t, val):
        tr = self.tree
        for (kind, opp), nodes in self.terms[t].items():
            at = torch.tensor(nodes, device=self.dev)
            pot = torch.tensor([float(tr.pot[x]) for x in nodes], dtype=torch.float64, device=self.dev)[:, None]
            bet = torch.tensor([float(tr.bets[x][t]) for x in nodes], dtype=torch.float64, device=self.dev)[:, None]
            r = [self.reach[o][at] for o in opp]
            if kind == "showdown":
                s = self.str[t]
                if len(opp) == 1:
                    free = (~self.share[t][opp[0]]).double()
                    so = self.str[opp[0]][None, :]
                    v = sum(c * (r[0] @ (free * m).T) for c, m in
                            ((pot - bet, so < s[:, None]), (pot / 2 - bet, so == s[:, None]), (-bet, so > s[:, None])))
                else:
                    v = torch.zeros(len(nodes), self.H[t], dtype=torch.float64, device=self.dev)
                    s1, s2 = self.str[opp[0]], self.str[opp[1]]
                    every = self.pairs(t, *opp, *r)
                    for g in torch.unique(s):
                        of = torch.nonzero(s == g)[:, 0]
                        part = lambda lo1, lo2: self.pairs(t, *opp, r[0] * (s1 < g if lo1 else s1 == g),  # noqa: E731
                                                           r[1] * (s2 < g if lo2 else s2 == g), of)
                        win, two, three = part(1, 1), part(0, 1) + part(1, 0), part(0, 0)
                        v[:, of] = ((pot - bet) * win + (pot / 2 - bet) * two + (pot / 3 - bet) * three -
                                    bet * (every[:, of] - win - two - three))
                    v = torch.where(every != 0, v, 0.0)
            else:
                if len(opp) == 1:
                    mass = r[0] @ (~self.share[t][opp[0]]).double().T
                else:
                    mass = self.pairs(t, *opp, *r)
                if kind == "leaf":
                    idx = torch.tensor([tr.leaf[x] for x in nodes], device=self.dev)
                    v = mass * self.leaf[idx, t, :self.H[t]]
                else:
                    won = torch.tensor([tr.player[x] == t for x in nodes], device=self.dev)[:, None]
                    v = mass * torch.where(won, pot - bet, -bet)
            val[at] = v

    def climb(self, t, val, sigma, best=False, ev=None):
        """Values of the decisions above val's terminals for traverser t."""
        for level in reversed(self.levels):
            for q, at in level:
                e = val[self.kids[at]]
                if q != t:
                    v = e.sum(1)
                elif best:
                    v = torch.where(self.legal[at][:, :, None], e, -math.inf).amax(1)
                else:
                    v = (sigma[at][:, :, :self.H[t]] * e).sum(1)
                    if ev is not None:
                        ev[at] = e
                val[self.dec_t[at]] = v

    def deal_mass(self):
        r = [w[None, :] for w in self.weight]
        m = r[1] @ (~self.share[0][1]).double().T if self.n == 2 else self.pairs(0, 1, 2, r[1], r[2])
        return float((self.weight[0] * m[0]).sum())

    def size(self):
        """Rows of the FP64 work per pass, to tell what would take long."""
        groups = sum(len(torch.unique(self.str[t])) for t in range(self.n)) if self.tree.river and self.n == 3 else 0
        return self.N * self.n * self.mh, groups


def _exact_solve(case, seed):
    if case["players"] > 3:
        return None      # three counted opponents: the sum over triples takes minutes
    g = _Game(case, seed)
    values, groups = g.size()
    if case["iterations"] * (1e-3 * g.n * len(g.levels) + 3e-10 * values + 4e-3 * groups) > 20:
        return None      # over about 20 seconds
    f64 = torch.float64
    A, mh = ssg.SS_MAX_ACTIONS, g.mh
    R = torch.zeros(len(g.dec), A, mh, dtype=f64, device=g.dev)
    S = torch.zeros_like(R)
    legal = g.legal[:, :, None]
    owned = [torch.tensor(g.owner == p, device=g.dev)[:, None, None] for p in range(g.n)]
    na = torch.tensor(g.na, dtype=f64, device=g.dev)[:, None, None]

    def match():
        pos = torch.clamp(R, min=0)
        s = pos.sum(1, keepdim=True)
        return torch.where(s > 0, pos / torch.where(s > 0, s, 1.0), 1.0 / na) * legal

    sigma = match()
    for p in range(g.n):
        g.set_reach(p, sigma)
    for it in range(1, case["iterations"] + 1):
        for t in range(g.n):
            root = sigma[0, :g.na[0], :g.H[g.owner[0]]].clone()
            val = torch.zeros(g.N + 1, g.H[t], dtype=f64, device=g.dev)
            ev = torch.zeros(len(g.dec), A, g.H[t], dtype=f64, device=g.dev)
            g.terminals(t, val)
            g.climb(t, val, sigma, ev=ev)
            pad = (0, mh - g.H[t])
            ev = torch.nn.functional.pad(ev, pad)
            v = torch.nn.functional.pad(val[g.dec_t], pad)[:, None, :]
            mine = owned[t] & legal
            S = torch.where(mine, S + it * sigma, S)
            R = torch.where(mine, (R + ev - v) * (it / (it + 1)), R)
            sigma = match()
            g.set_reach(t, sigma)
    s = S.sum(1, keepdim=True)
    avg = torch.where(s > 0, S / torch.where(s > 0, s, 1.0), 1.0 / na) * legal
    for p in range(g.n):
        avg[torch.tensor(g.owner == p, device=g.dev), :, g.H[p]:] = 0.0
    last = torch.zeros(mh, dtype=f64, device=g.dev)
    last[:g.H[g.n - 1]] = val[0]
    # regret matching amplifies rounding: the last iterate (no average) follows it after tens of
    # iterations, a near-tie's average after many hundreds, and 64 bits then play another near-equilibrium
    return {"avg": avg if case["iterations"] <= 300 else None, "root": root if case["iterations"] <= 30 else None,
            "ev": last}


def _exact_exploit(case, seed):
    g = _Game(case, seed)
    profile = torch.tensor(_profile(g.na, g.owner, g.H, g.mh, seed), device=g.dev).double()
    for p in range(g.n):
        g.set_reach(p, profile)
    br, cur = [], []
    for t in range(g.n):
        val = torch.zeros(g.N + 1, g.H[t], dtype=torch.float64, device=g.dev)
        g.terminals(t, val)
        for best, to in ((False, cur), (True, br)):
            g.climb(t, val, profile, best=best)
            to.append(float((g.weight[t] * val[0]).sum()))
    z = g.deal_mass()
    nash = (sum(br) - sum(cur)) / z
    return {"pct": nash / g.n / case["pot"] * 100, "nash": nash, "br": np.array(br), "cur": np.array(cur), "mass": z}


_FOLD, _FACTOR = (0.0, 0.35, 0.0, 0.0), (1.0, 0.7, 1.0, 1.4)


def _sampled(cards, seed, large):
    return sorted(int(c) for c in np.random.RandomState(seed).choice(cards, 12, replace=False)) if large else cards


def _exact_leaves(case, seed):
    """Share of up to 2000 opponent hand tuples that each hand beats, averaged
    over the runouts, then the bias adjustment of every continuation profile."""
    board, hands, _ = _board_and_ranges(case, seed)
    n, H = case["players"], [len(h) for h in hands]
    mh, large = max(H), max(H) > 50
    first = _sampled([c for c in range(52) if c not in board], 42, large)
    runouts = ([[c] for c in first] if case["board"] == 4 else
               [[c, d] for c in first
                for d in _sampled([x for x in range(52) if x not in board and x != c], 43 + c, large)])
    bits = [(np.uint64(1) << h[:, 0].astype(np.uint64)) | (np.uint64(1) << h[:, 1].astype(np.uint64)) for h in hands]
    if len(runouts) * n * mh * min(2000.0, float(mh) ** (n - 1)) > 1.2e9:
        return None      # over about 20 seconds
    raw, cnt = np.zeros((n, mh)), np.zeros((n, mh))
    for more in runouts:
        st = [_strengths(board + more, h) for h in hands]
        live = [np.flatnonzero(s > 0) for s in st]
        for p in range(n):
            opp = [q for q in range(n) if q != p]
            if not len(live[p]) or any(not len(live[q]) for q in opp):
                continue
            if math.prod(len(live[q]) for q in opp) <= 2000:
                tup = np.array(list(itertools.product(*(live[q] for q in opp))))
            else:
                rng = random.Random(42)
                lists = [live[q].tolist() for q in opp]
                tup = np.array([[rng.choice(x) for x in lists] for _ in range(2000)])
            mask, clash = np.zeros(len(tup), np.uint64), np.zeros(len(tup), bool)
            for k, q in enumerate(opp):
                clash |= (mask & bits[q][tup[:, k]]) != 0
                mask |= bits[q][tup[:, k]]
            so = np.stack([st[q][tup[:, k]] for k, q in enumerate(opp)])
            best = so.max(0)
            ties = (so == best).sum(0)
            hs = st[p][live[p]][:, None]
            free = ((bits[p][live[p]][:, None] & mask) == 0) & ~clash
            won = np.where(hs > best, 1.0, np.where(hs == best, 1.0 / (1.0 + ties), 0.0)) * free
            valid = free.sum(1)
            ok = valid > 0
            raw[p, live[p][ok]] += won.sum(1)[ok] / valid[ok]
            cnt[p, live[p][ok]] += 1
    eq = np.where(cnt > 0, raw / np.maximum(cnt, 1), 0.0)
    tree = _Tree(case)
    per = 4 ** n
    out = np.zeros((len(tree.chain_heads) * per, n, mh))
    for first_leaf, pot in tree.chain_heads:
        for combo in range(per):
            row = first_leaf // per * per + combo
            if row >= len(out):
                continue
            prof = [(combo // 4 ** i) % 4 for i in range(n)]
            for p in range(n):
                other = max(0, min(3, int(round(sum(prof[q] for q in range(n) if q != p) / (n - 1)))))
                e = eq[p, :H[p]]
                out[row, p, :H[p]] = (_FOLD[other] * 0.5 * pot +
                                      (1.0 - _FOLD[other]) * (e - 0.5) * pot * _FACTOR[prof[p]] * _FACTOR[other])
    return out


def exact(case, seed):
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "exploit":
        return _exact_exploit(case, seed)
    if case["kind"] == "leaves":
        return _exact_leaves(case, seed)
    return None      # batches and flop-to-river trees: minutes in 64 bits

"""The multi-street solver on a caller's trees from the turn or the river on:
few terminals (a block each) and many on few boards (a warp each, several blocks
to a board), around the lines between the forms.  Every node's value after one
iteration against the FP64 restatement, with the tolerance of
test_flop_terminals_gpu.py, whose reasons hold here (fewer levels).  A terminal
value of a hand that no opponent hand of positive weight is compatible with is
exactly 0.  (Not every exact 0 of the restatement: the last traverser meets the
other's strategy of this iteration, where a regret that cancels in FP64 can be
1e-9 in FP32 and give a hand reach.)"""
import ctypes

import numpy as np
import pytest

import flop_solve as fsm
import street_solver_gpu as ssg

pytestmark = pytest.mark.gpu


def betting_tree(board, streets, raises, sizes, pot=100, stack=9000):
    """Check, call, fold and raises of the given pot sizes; a call before the
    river leads to a chance node over every card left."""
    nodes = []

    def new():
        nodes.append(None)
        return len(nodes) - 1

    def put(x, kind, player, kids, pot, bets, brd):
        nodes[x] = (kind, player, kids, pot, bets, brd)

    def decide(x, player, bets, pot, left, brd, checked):
        need, kids = bets[1 - player] - bets[player], []
        moves = [("fold", 0)] if need > 0 else []
        moves.append(("call", 0))
        if left > 0:
            to = [bets[1 - player] + max(1, round((pot + need) * z)) for z in sizes]
            moves += [("raise", t) for t in to if t < stack]
        for move, to in moves:
            y = new()
            kids.append(y)
            b = list(bets)
            if move == "fold":
                put(y, fsm.NODE_FOLD, 1 - player, [], pot, b, brd)
            elif move == "raise":
                b[player] = to
                decide(y, 1 - player, b, pot + to - bets[player], left - 1, brd, False)
            else:
                b[player] = bets[1 - player]
                if not checked and need == 0:
                    decide(y, 1 - player, b, pot, left, brd, True)
                elif len(brd) == 5:
                    put(y, fsm.NODE_SHOWDOWN, -1, [], pot + need, b, brd)
                else:
                    deals = []
                    for c in range(52):
                        if c not in brd:
                            z = new()
                            deals.append(z)
                            decide(z, 0, b, pot + need, streets[1], brd + [c], False)
                    put(y, fsm.NODE_CHANCE, -1, deals, pot + need, b, brd)
        put(x, fsm.NODE_DECISION, player, kids, pot, list(bets), brd)

    decide(new(), 0, [0, 0], pot, raises, list(board), False)
    return nodes


def subgame(nodes, hands, weights):
    rows, ch, depth = (fsm.FSNode * len(nodes))(), [], np.zeros(len(nodes), np.int32)
    for i, (kind, player, kids, pot, bets, brd) in enumerate(nodes):
        r = [kind, player, len(kids), len(ch), pot, *bets, *(brd + [0] * 5)[:5], len(brd)]
        ch.extend(kids)
        for k in kids:
            depth[k] = depth[i] + 1      # (a parent is numbered before its children)
        ctypes.memmove(ctypes.byref(rows[i]), (ctypes.c_int * 13)(*r), 52)
    sg = object.__new__(fsm.FlopSubgame)
    sg.lib, sg.td, sg.nh = fsm.bind(ssg.load_library(200)), fsm.FSTreeData(), [len(h) for h in hands]
    children = (ctypes.c_int * len(ch))(*ch)
    sg.keep = rows, children
    sg.td.nodes, sg.td.children = ctypes.cast(rows, ctypes.POINTER(fsm.FSNode)), ctypes.cast(children, ctypes.POINTER(ctypes.c_int))
    sg.td.num_nodes, sg.td.num_children_total = len(nodes), len(ch)
    for p in range(2):
        sg.td.num_hands[p] = len(hands[p])
        for i, (h, w) in enumerate(zip(hands[p], weights[p])):
            sg.td.hands[p][i][0], sg.td.hands[p][i][1], sg.td.weights[p][i] = int(h[0]), int(h[1]), float(w)
    flat = np.frombuffer(rows, np.int32).reshape(-1, 13).copy()
    return sg, flat, np.array(ch, np.int32), depth


@pytest.mark.parametrize("cards,raises,streets,sizes,n0,n1,repeat,folds,showdowns", [
    (5, 1, (), [0.75], 33, 20, False, (1, 296), (1, 4096)),
    (5, 4, (), [0.33, 0.75, 1.5], 40, 200, False, (1, 296), (1, 4096)),
    (5, 6, (), [0.33, 0.75, 1.5], 24, 25, True, (297, 10**6), (1, 4096)),
    (5, 6, (), [0.2, 0.4, 0.6, 0.8], 25, 24, False, (297, 10**6), (4097, 10**6)),
    (4, 1, (0, 1), [0.75], 30, 31, True, (1, 296), (1, 4096)),
    (4, 3, (0, 2), [0.5, 1.0], 20, 33, False, (297, 10**6), (4097, 10**6)),
])
def test_values_after_one_iteration(cards, raises, streets, sizes, n0, n1, repeat, folds, showdowns):
    from oracle.oracle import FlopOracle
    rng = np.random.default_rng(cards * 100 + raises)
    board = [int(c) for c in rng.permutation(52)[:cards]]
    nodes = betting_tree(board, streets, raises, sizes)
    kinds = [n[0] for n in nodes]
    assert folds[0] <= kinds.count(fsm.NODE_FOLD) <= folds[1], kinds.count(fsm.NODE_FOLD)
    assert showdowns[0] <= kinds.count(fsm.NODE_SHOWDOWN) <= showdowns[1], kinds.count(fsm.NODE_SHOWDOWN)
    combos = [(a, b) for a in range(52) for b in range(a + 1, 52)]   # some touch the board
    hands, weights = [], []
    for n in (n0, n1):
        h = np.array([combos[i] for i in rng.choice(len(combos), n, replace=False)], np.int32)
        if repeat:
            h[-3:] = h[:3]
        w = rng.uniform(0.1, 1.0, n).astype(np.float32)
        w[rng.random(n) < 0.2] = 0.0
        hands.append(h)
        weights.append(w)
    sg, flat, ch, depth = subgame(nodes, hands, weights)
    got = sg.solve(1, extract=True)
    H, W = np.zeros((2, 200, 2), np.int32), np.zeros((2, 200), np.float32)
    for p in range(2):
        H[p, :len(hands[p])], W[p, :len(hands[p])] = hands[p], weights[p]
    ref = FlopOracle().solve(flat, ch, depth, int(depth.max()), H, W, np.array([n0, n1], np.int32), 1, "f64")
    a, b = got["all_cfv"], ref["all_cfv"]
    assert np.abs(a - b).max() <= 1e-4 * max(np.abs(b).max(), 1e-30)
    masks = [[1 << int(h[0]) | 1 << int(h[1]) for h in x] for x in hands]
    none = {}   # board -> the last traverser's hands without a compatible opponent hand
    for x in np.flatnonzero((flat[:, 0] == fsm.NODE_FOLD) | (flat[:, 0] == fsm.NODE_SHOWDOWN)):
        brd = 0
        for c in flat[x, 7:7 + flat[x, 12]]:
            brd |= 1 << int(c)
        if brd not in none:
            live = [m for m, w in zip(masks[0], weights[0]) if w > 0 and not m & brd]
            none[brd] = np.array([not any(not m & o for o in live) for m in masks[1]])
        assert np.all(a[x, :n1][none[brd]] == 0)

"""Four-way showdowns (k_term_sd3) where its splits have edges: ranges whose
hands leave blocks of 256 rank positions empty or crowd into one, a number of
hands on each side of a lane split, tie groups across block ends (fewer and
more positions than warps), and a third opponent with one live hand.  Against
the oracle's tuple enumeration, test_parity_gpu's tolerances."""
import numpy as np
import pytest

import workloads as wl
from cards import card_to_int
from test_cr3_gpu import oracle_f32
from test_parity_gpu import solve, strict

QUADS = ["Ks", "Kd", "Kh", "Kc", "2s"]   # a hand ranks by its best card: 12 tie groups of 4 to 200 positions
ROYAL = ["As", "Ks", "Qs", "Js", "Ts"]   # one tie group of all positions
PLAIN = ["2c", "7d", "9h", "Js", "Qd"]


def subgame(seed, board, sizes, ace=(), single=None):
    """sizes: hands per player; ace: players who hold only hands with an ace;
    single: the player of whose hands one has weight."""
    cfg = wl.config("river6", seed=seed, num_players=4, bet_sizes=[1.0], max_raises=1)
    cfg["board"] = [card_to_int(c) for c in board]
    rng = np.random.default_rng(seed)
    hands, weights = wl.make_ranges(rng, cfg["board"], 4)
    aces = {card_to_int(r) for r in ("As", "Ad", "Ah", "Ac")}
    for p, n in enumerate(sizes):
        ok = [i for i, h in enumerate(hands[p]) if p not in ace or aces & {int(h[0]), int(h[1])}]
        sel = np.sort(rng.choice(ok, n, replace=False))
        hands[p], weights[p] = hands[p][sel], weights[p][sel]
        if p == single:
            weights[p][np.arange(n) != n // 2] = 0.0
    cfg["hands"], cfg["weights"] = hands, weights
    return cfg


@pytest.mark.gpu
@pytest.mark.parametrize("seed,board,sizes,ace,single", [
    (91, PLAIN, (16, 17, 33, 24), (), None),
    (92, QUADS, (16, 33, 16, 20), (0,), None),      # the first player's hands all in the top group
    (93, QUADS, (40, 16, 18, 16), (0, 2), 3),       # 40 hands in one block; one live hand
    (94, ROYAL, (65, 16, 16, 16), (), None),        # the 65 hands spread over every block
    (95, PLAIN, (16, 16, 16, 130), (), 1),
])
def test_four_way_showdowns_against_oracle(oracle, seed, board, sizes, ace, single):
    cfg = subgame(seed, board, sizes, ace, single)
    ours, lv = solve(cfg, 3)
    strict(ours, oracle_f32(oracle, cfg, 3, lv))

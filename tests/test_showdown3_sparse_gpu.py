"""Three-way showdowns with few live hands (k_term_sd2's sparse form): at the
line against the general form, and where an opponent has almost no hands, or
the hands tie in long groups, against the FP64 oracle.

A range just above the rule's line takes the general form; here it is the
sparse form's range with a few hands of weight 1e-30 added.  Where every hand
meets opponents' hands of total weight of order 1, those enter FP64 sums of
order 1, so the other hands' values round to the same floats, or at worst to a
neighbour (6e-8 relative, a handful of iterations of regrets): 1e-5 on
probabilities is far above that and far below a lost or doubled hand (1 / 400
of a mass).  Against the oracle: test_parity_gpu's tolerances."""
import numpy as np
import pytest

import workloads as wl
from cards import card_to_int
from test_parity_gpu import oracle_pair, solve, strict

LINE = 400   # live hands up to which the sparse form is taken


def ranges(seed, live, board, tiny):
    """Per player `live` hands with weight, and with tiny more hands of weight
    1e-30 up to LINE + 1; the same hands for each value of tiny."""
    cfg = wl.config("river6", seed=seed, num_players=3)
    if board is not None:
        cfg["board"] = [card_to_int(c) for c in board]
    rng = np.random.default_rng(seed)
    hands, weights = wl.make_ranges(rng, cfg["board"], 3, LINE + 1)
    for p in range(3):
        keep = rng.permutation(LINE + 1) < live[p]
        weights[p] = np.where(keep, 0.05 + weights[p], 1e-30 if tiny else 0.0).astype(np.float32)
    cfg["hands"], cfg["weights"] = hands, weights
    return cfg


@pytest.mark.gpu
@pytest.mark.parametrize("seed,live,board", [
    (81, (400, 400, 400), None),                          # the last range of the sparse form
    (84, (20, 120, 60), ["As", "Ks", "Qs", "Js", "Ts"]),  # one group over all positions
])
def test_sparse_form_gives_the_general_forms_values(seed, live, board):
    a, _ = solve(ranges(seed, live, board, False), 3)
    cfg = ranges(seed, live, board, True)
    b, _ = solve(cfg, 3)
    assert np.isfinite(a["root_ev"]).all()
    w = np.asarray(cfg["weights"][a["root_player"]]) > 1e-20
    ra, rb = np.asarray(a["root_strategy"]), np.asarray(b["root_strategy"])
    assert ra.shape == rb.shape
    n = len(w)
    ra, rb = ra.reshape(-1, n), rb.reshape(-1, n)
    np.testing.assert_allclose(ra[:, w], rb[:, w], rtol=0, atol=1e-5)
    ea, eb = np.asarray(a["root_ev"], np.float64), np.asarray(b["root_ev"], np.float64)
    assert np.abs(ea - eb).max() <= 1e-5 * np.abs(ea).max(), (ea, eb)


@pytest.mark.gpu
@pytest.mark.parametrize("seed,live,board", [
    (82, (7, 33, 400), None),                             # groups without one or both opponents
    (83, (64, 65, 31), ["Ks", "Kd", "Kh", "Kc", "2s"]),   # long tie groups, several mask words
])
def test_sparse_form_against_oracle(oracle, seed, live, board):
    cfg = ranges(seed, live, board, False)
    for p in range(3):   # the oracle's time goes by hands, with weight or without
        keep = cfg["weights"][p] > 0
        cfg["hands"][p], cfg["weights"][p] = cfg["hands"][p][keep], cfg["weights"][p][keep]
    ours, lv = solve(cfg, 3)
    _, r64 = oracle_pair(oracle, cfg, 3, lv)
    strict(ours, r64)

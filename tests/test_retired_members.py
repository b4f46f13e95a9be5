"""A member that has left a batch keeps its items in the captured launches
while its own tables are already freed, so a merged kernel asks whether the
member is live before it reads anything of the member's.

On CPU the order is read from the kernels' source: in every function that
takes the array of contexts, the question comes before the first load through
a member's pointers.  On the GPU a server retires small members under a large
one that keeps iterating, with a memory pool that gives freed pages back, and
the large member's result is its solo result."""
import ctypes
import os
import re

import numpy as np
import pytest

import workloads as wl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "poker-solver_b200", "csrc")

# loads through a member's pointers, or helpers that form them for one
LOADS = re.compile(r"__ldg\((?!&?items|heads)|reach_rows|val_rows|cr2_view|cfv_view|cp_async|\bc\.(?!H\b|dup\b|sd_span\b)\w+\[|\br\[")
ASKS = re.compile(r"retired\(ctxs|\.live\b")


def merged_functions():
    for name in ("ss_kernels.cu", "ss_cr2_tc.cuh"):
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"^__(?:global|device)__[^;{]*?\b(k_\w+|\w+_terminal|retired)\(([^;{]*?)\)\s*\{(.*?)^\}", src,
                             re.M | re.S):
            if re.search(r"const DevCtx \*__restrict__ ctxs", m.group(2)):
                yield m.group(1), m.group(3)


def test_merged_kernels_ask_first():
    seen = []
    for name, body in merged_functions():
        ask, load = ASKS.search(body), LOADS.search(body)
        if ask is None:
            # a kernel around one that asks
            assert load is None and re.search(r"(sd1|cr1)_terminal<", body), name
            continue
        assert load is None or ask.start() < load.start(), name
        seen.append(name)
    assert {"sd1_terminal", "cr1_terminal", "k_reach", "k_cfv", "k_term_fill", "k_term_cr1_dup", "k_term_cr2",
            "k_term_sd2", "k_term_enum", "k_term_cr3", "k_term_sd3", "k_avg_many", "k_br_reach_many",
            "k_br_value_many", "k_br_root_many", "k_bump_many", "k_snapshot_many", "k_term_cr2_tc"} <= set(seen), seen


class NoCachedPages:
    """The device's default memory pool gives freed pages back (release
    threshold 0) inside the block."""

    def __enter__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        dev, self.pool = ctypes.c_int(), ctypes.c_void_p()
        assert self.cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), dev) == 0
        self.was = ctypes.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, 4, ctypes.byref(self.was)) == 0   # release threshold
        self.set(0)

    def set(self, n):
        v = ctypes.c_uint64(n)
        assert self.cu.cuMemPoolSetAttribute(self.pool, 4, ctypes.byref(v)) == 0

    def __exit__(self, *a):
        self.set(self.was.value)


@pytest.mark.gpu
def test_server_iterates_past_released_members():
    def river(seed, **over):
        cfg = wl.config("hu_river", seed=seed, **over)
        return wl.AbiSubgame(cfg, max_hands=1326)

    big = river(61, bet_sizes=[0.33, 0.75, 1.5], max_raises=3, num_hands=1081)
    small = [river(62 + i, bet_sizes=[1.0], max_raises=1, num_hands=60 + 200 * i) for i in range(3)]
    subs = [big] + small
    lib = big.lib
    kw = dict(block_iterations=10, target_exploitability=0.3, max_iterations=400)
    alone = []
    for sg in subs:
        srv = wl.Server(lib, **kw)
        alone.append(srv.wait(srv.submit(sg), sg.nh))
        srv.close()
    its = [a["stats"]["iterations_run"] for a in alone]
    assert min(its[1:]) < its[0], its   # members leave while the large one goes on
    with NoCachedPages():
        srv = wl.Server(lib, **kw)
        ids = [srv.submit(sg) for sg in subs]
        mixed = [srv.wait(i, sg.nh) for i, sg in zip(ids, subs)]
        srv.close()
    for a, m in zip(alone, mixed):
        for k in ("root_strategy", "root_ev", "avg_strategies", "avg_node_ids"):
            assert np.array_equal(a[k], m[k]), k
        assert a["stats"]["iterations_run"] == m["stats"]["iterations_run"]
    for sg in subs:
        sg.free()


def test_small_solve_stops_block_by_block():
    """k_small_solve waits at barriers that count threads, so whatever makes it
    return before them is decided once for the block: its early returns follow a
    block-wide vote or a grid barrier's shared answer."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "ss_kernels.cu")).read())
    body = re.search(r"k_small_solve\(const __grid_constant__.*?\{(.*?)^\}", src, re.M | re.S).group(1)
    returns = [line.strip() for line in body.split("\n") if re.search(r"\breturn;", line)]
    assert returns and all("__syncthreads_or(" in r or "grid_barrier(" in r for r in returns), returns

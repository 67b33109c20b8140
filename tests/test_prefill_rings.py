"""The operand rings of the prefill kernel, walked on the CPU with the kernel's constants.

A block serves two query heads of one kv-head from one ring of K tiles and one ring of V tiles; a vertical-line tile
belongs to one head and is handed back by the other.  The waits of the producer and of the two issuing warps are
replayed here for every pair of tile counts: a set of waits that wait for one another would show as a state in which
nobody can go on."""

import itertools
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyquant_b200", "csrc", "hq_prefill_tc.cu")


def constant(name):
    with open(SOURCE) as f:
        return int(re.search(r"constexpr int %s = (\d+);" % name, f.read()).group(1))


K_DEPTH, V_DEPTH, NEAR = constant("kKStages"), constant("kVStages"), constant("kNearRun")


def ring_items(n_rest, nv, n_win):
    """Owner of every item in load order: 2 = both heads, else the head of a vertical-line tile."""
    vert = [h for j in range(max(nv)) for h in (0, 1) if j < nv[h]]
    return [2] * n_rest + vert + [2] * n_win


def issue_order(items, h, near):
    """The waits and hand-overs of head h's issuing warp, in program order.  ``near``: the longest run of the other head's
    items behind which a Q K^T may be waited for before the P V that is due (None: whatever the run)."""
    ops, k, v = [], 0, 0
    feeds = lambda i: items[i] in (2, h)                                     # noqa: E731
    n_t = sum(feeds(i) for i in range(len(items)))

    def run_ahead():
        n = 0
        while k + n < len(items) and not feeds(k + n):
            n += 1
        return near is not None and n > near

    def k_ready():
        nonlocal k
        while True:
            ops.append(("wait_k", k))
            if feeds(k):
                return
            ops.append(("free_k", k))
            k += 1

    def qk():
        nonlocal k, issued
        ops.extend([("qk", issued), ("free_k", k)])
        k += 1
        issued += 1

    issued = 0
    for t in range(n_t):
        if issued == t:
            while not feeds(k):
                assert k == v
                ops.extend([("wait_k", k), ("free_k", k), ("wait_v", v), ("free_v", v)])
                k, v = k + 1, v + 1
            for i in range(2):
                if issued < n_t and (i == 0 or not run_ahead()):
                    k_ready()
                    qk()
        more = issued == t + 2 and issued < n_t and not run_ahead()
        while True:
            ops.append(("wait_v", v))
            if feeds(v):
                break
            ops.append(("free_v", v))
            v += 1
        if more:
            k_ready()
        ops.extend([("wait_p", t), ("pv", t), ("free_v", v)])
        v += 1
        if more:
            qk()
    assert k == v == len(items) and issued == n_t
    return ops


def carries(items, programs, k_depth=K_DEPTH, v_depth=V_DEPTH):
    """Run the producer and the issuing warps as far as they go; True if all of them finish."""
    n = len(items)
    loaded = {"k": 0, "v": 0}
    freed = {"k": [0] * n, "v": [0] * n}
    pc, qk, pv = [0] * len(programs), [0] * len(programs), [0] * len(programs)
    while True:
        moved = False
        for ring, depth in (("k", k_depth), ("v", v_depth)):
            i = loaded[ring]
            while i < n and (i < depth or freed[ring][i - depth] == len(programs)):
                i, moved = i + 1, True
            loaded[ring] = i
        for h, ops in enumerate(programs):
            while pc[h] < len(ops):
                op, x = ops[pc[h]]
                if op in ("wait_k", "wait_v"):
                    if x >= loaded[op[-1]]:
                        break
                elif op in ("free_k", "free_v"):
                    freed[op[-1]][x] += 1
                elif op == "qk":
                    qk[h] = x + 1
                elif op == "wait_p":
                    # the softmax warps: scores of the tile, and (to move the reference) every P V before it
                    if not (qk[h] > x and pv[h] >= x):
                        break
                else:
                    pv[h] = x + 1
                pc[h] += 1
                moved = True
        if all(pc[h] == len(ops) for h, ops in enumerate(programs)):
            return True
        if not moved:
            return False


COUNTS = [(a, b) for a in range(15) for b in range(15)] + [(0, 40), (40, 0), (3, 33), (33, 3), (17, 40), (40, 17), (39, 40)]


@pytest.mark.parametrize("n_rest", [0, 1, 2, 3, 5, 20])
def test_rings_carry_every_pair_of_tile_counts(n_rest):
    for nv, n_win in itertools.product(COUNTS, (1, 2, 3, 4, 7)):
        items = ring_items(n_rest, nv, n_win)
        programs = [issue_order(items, h, NEAR) for h in (0, 1)]
        assert carries(items, programs), (n_rest, nv, n_win)
        # one slot less in either ring still carries them: the waits do not live on the last slot
        assert carries(items, programs, v_depth=V_DEPTH - 1), (n_rest, nv, n_win)


@pytest.mark.parametrize("n_rest,nv,n_win", [(20, (0, 7), 4), (20, (7, 0), 4), (20, (3, 8), 4), (20, (5, 10), 4), (20, (10, 15), 4)])
def test_the_walk_finds_waits_that_close_a_circle(n_rest, nv, n_win):
    """The order that waits for K of tile t + 2 before P V of t whatever lies between: stuck on these counts."""
    items = ring_items(n_rest, nv, n_win)
    assert not carries(items, [issue_order(items, h, None) for h in (0, 1)])


def test_a_single_head_block_never_waits_for_a_neighbour():
    for n_rest, n, n_win in itertools.product((0, 1, 20), (0, 1, 9), (1, 4)):
        items = ring_items(n_rest, (n, 0), n_win)
        assert carries(items, [issue_order(items, 0, NEAR)])

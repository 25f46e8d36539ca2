"""Barriers between the passes of factored programs, on CPU: a walk over the planned
tables with the barriers of the kernels that run them.  A pass flagged as one of a
phase ends with a warp barrier, every other one with a barrier over the register's
threads, whether it has anything to do or not; no warp may then read or write a
slot that another one has written, or write one that another one has read, since
the last barrier over all of them."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.test_plan import HDR, lib  # noqa: F401
from tests.test_plan_factored import LIST, PASS, one_qubit_ops, plan

WARP = 2  # DK_PASS_WARP
STORE = 4  # DK_FX_STORE


def hazards(blob, prec, idle_barrier=True, conds_on=0):
    """Accesses of one tile across warps without a barrier between them.
    `idle_barrier`: passes with nothing to do keep their barrier; `conds_on`: the
    tile conditions that hold, a bit each."""
    h = np.frombuffer(blob, HDR, 1)[0]
    m = int(h["m"])
    passes = np.frombuffer(blob, PASS, int(h["npass"]), int(h["pass_off"]))
    nlist = max(int(p["list"]) + (1 << (int(p["cond"]) >> 15)) for p in passes)
    lists = np.frombuffer(blob, LIST, nlist, int(h["pass_off"]) + PASS.itemsize * len(passes))
    amp = 16 if prec == 2 else 8
    tid = np.arange(1 << (m - 4))
    if len(tid) <= 32:
        return 0
    warp, reg = np.broadcast_to((tid >> 5)[:, None], (len(tid), 16)), np.arange(16)
    writer = np.full(1 << m, -1)  # since the last barrier over all warps
    reader = np.full(1 << m, -1)
    several = np.zeros(1 << m, dtype=bool)  # read by more than one warp
    found = 0
    for p in passes:
        v = 0
        for c in range(int(p["cond"]) >> 15):
            v |= ((conds_on >> ((int(p["cond"]) >> (5 * c)) & 31)) & 1) << c
        li = lists[int(p["list"]) + v]
        idle = bool(li["idle"]) and not int(p["flags"]) & STORE
        if not idle:
            sg = (p["slo"][tid & 31].astype(np.int64) ^ p["shi"][tid >> 5]) // amp
            for gat in (True, False):
                vec = li["gt"] if gat else li["st"]
                off = int(li["gc"] if gat else li["sc"]) // amp
                sl = sg[:, None] ^ off ^ np.bitwise_xor.reduce(
                    [np.where((reg >> j) & 1, int(vec[j]) // amp, 0) for j in range(4)])[None, :]
                w = writer[sl]
                found += int(((w >= 0) & (w != warp)).sum())
                if gat:
                    r = reader[sl]
                    several[sl] |= (r >= 0) & (r != warp)
                    reader[sl] = warp
                else:
                    r = reader[sl]
                    found += int((several[sl] | ((r >= 0) & (r != warp))).sum())
                    writer[sl] = warp
        if int(p["flags"]) & WARP or (idle and not idle_barrier):
            continue
        writer[:], reader[:], several[:] = -1, -1, False
    return found


def phases_of_angle_0(n, seed):
    """Layers of one-qubit gates and of controlled phases between all pairs, all of
    angle 0: a parametrised circuit before its first step."""
    rng = W.rng_for(seed)
    ops = []
    for _ in range(3):
        ops += [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q]) for q in range(n)]
        pairs = [(int(a), int(b)) for a in range(n) for b in range(a)]
        rng.shuffle(pairs)
        ops += [W.Op(np.diag([1, 1]).astype(complex), [a], {b}) for a, b in pairs]
    return ops


def equal_pairs(n, seed):
    """CNOTs that undo each other among one-qubit gates."""
    rng = W.rng_for(seed)
    ops = []
    for _ in range(40):
        if rng.random() < 0.4:
            ops.append(W.Op(W.u3(*rng.uniform(0, 6, 3)), [int(rng.integers(n))]))
        a, b = (int(x) for x in rng.permutation(n)[:2])
        ops += [W.Op(W.X.copy(), [a], {b})] * 2
    return ops


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n", [10, 11, 12])
def test_one_tile(lib, n, prec):  # noqa: F811
    lost = 0
    for seed in range(12):
        for ops in (phases_of_angle_0(n, seed), equal_pairs(n, seed),
                    one_qubit_ops(W.rng_for(seed), n, 80)):
            for _, blob, _, _ in plan(lib, ops, n, prec):
                assert hazards(blob, prec) == 0
                lost += hazards(blob, prec, idle_barrier=False) > 0
    assert lost > 0  # the circuits have idle passes whose barriers count


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n,tile_bits", [(14, None), (16, 11), (15, 10)])
def test_tiles_with_conditions(lib, n, tile_bits, prec):  # noqa: F811
    """A tile on which none, all or some of the conditions hold."""
    for seed in range(4):
        ops = phases_of_angle_0(n, seed)[:120] + one_qubit_ops(W.rng_for(seed), n, 80)
        for _, blob, _, _ in plan(lib, ops, n, prec, tile_bits):
            for on in (0, 0xffffffff, 0x55555555, 0x33333333):
                assert hazards(blob, prec, conds_on=on) == 0

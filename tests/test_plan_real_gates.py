"""Factored sweeps of gates whose factors share a stage, on CPU: rotations by real
angles and real matrices have no phases between them, so that many of them come into
one stage with the CNOTs in between as relabellings, along directions of one and of
several register bits.  Replayed against the gates one by one in extended
precision."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.test_plan import lib  # noqa: F401
from tests.test_plan_factored import run


def ry(t):
    return W.u3(t, 0, 0)


def apply_all(psi, ops):
    out, idx = psi.astype(np.clongdouble), np.arange(psi.size)
    for op in ops:
        on = np.ones(psi.size, dtype=bool)
        for c in op.controls:
            on &= (idx >> c) & 1 == 1
        for c in op.anticontrols:
            on &= (idx >> c) & 1 == 0
        t, m = op.targets[0], np.asarray(op.gate).astype(np.clongdouble)
        i0 = idx[on & ((idx >> t) & 1 == 0)]
        i1 = i0 | (1 << t)
        a, b = out[i0].copy(), out[i1].copy()
        out[i0], out[i1] = m[0, 0] * a + m[0, 1] * b, m[1, 0] * a + m[1, 1] * b
    return out


def check(lib, n, ops, seed, prec=2, tile_bits=None):  # noqa: F811
    rng = W.rng_for(seed)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    want = apply_all(psi, ops)
    got, _ = run(lib, ops, n, psi, prec, tile_bits)
    size = np.sqrt(float((np.abs(want) ** 2).sum()))
    err = np.sqrt(float((np.abs(got - want) ** 2).sum())) / size
    # real gates with condition numbers below 40, 150 of them at most: roundings of
    # 2^-53 (2^-24) each that grow by as much at worst; wrong orders are off by 1e-2
    assert err < (1e-12 if prec == 2 else 1e-4), float(err)


def test_rotations_on_both_sides_of_a_cnot(lib):  # noqa: F811
    """The control's rotation turns the direction of the target's second one."""
    for c, t, other in ((0, 3, 1), (3, 0, 1), (1, 2, 0), (2, 1, 3)):
        for ctl in ({"controls": {c}}, {"anticontrols": {c}}):
            x = W.Op(W.X.copy(), [t], ctl.get("controls", set()), ctl.get("anticontrols", set()))
            ops = [W.Op(ry(0.7), [c]), x, W.Op(ry(1.1), [t]), W.Op(ry(0.4), [other])]
            check(lib, 4, ops, 1)
            check(lib, 6, ops + ops[::-1], 2)


@pytest.mark.parametrize("prec,tile_bits", [(2, None), (1, None), (2, 5), (1, 4)])
def test_random_real_circuits(lib, prec, tile_bits):  # noqa: F811
    for seed in range(60):
        rng = W.rng_for(8700 + seed)
        n = int(rng.integers(4, 8)) if tile_bits is None else int(rng.integers(6, 9))
        ops = []
        for _ in range(int(rng.integers(10, 150))):
            q = [int(x) for x in rng.permutation(n)]
            r = rng.random()
            if r < 0.45:
                ops.append(W.Op(ry(rng.uniform(0, 6)), q[:1]))
            elif r < 0.75:
                anti = rng.random() < 0.3
                ops.append(W.Op(W.X.copy(), q[:1], set() if anti else {q[1]},
                                {q[1]} if anti else set()))
            elif r < 0.8:
                ops.append(W.Op(W.X.copy(), q[:1], set(q[1:3])))
            elif r < 0.86:
                ops.append(W.Op(ry(rng.uniform(0, 6)), q[:1], {q[1]}))
            elif r < 0.9:
                ops.append(W.Op(W.H.copy(), q[:1]))
            elif r < 0.94:
                ops.append(W.Op(np.array([[1, rng.uniform(-1, 1)], [0, 1]], dtype=complex), q[:1]))
            else:
                ops.append(W.Op(W.Z.copy(), q[:1], {q[1]} if rng.random() < 0.5 else set()))
        check(lib, n, ops, 8800 + seed, prec, tile_bits)


@pytest.mark.parametrize("entangler", ["chain", "ring", "all", "reverse"])
def test_real_ansatz(lib, entangler):  # noqa: F811
    """Layers of Ry and CNOTs, as variational circuits have them."""
    n = 6
    pairs = {"chain": [(q, q + 1) for q in range(n - 1)],
             "ring": [(q, (q + 1) % n) for q in range(n)],
             "all": [(a, b) for a in range(n) for b in range(a + 1, n)],
             "reverse": [(q + 1, q) for q in reversed(range(n - 1))]}[entangler]
    for seed in range(10):
        rng = W.rng_for(8900 + seed)
        ops = []
        for _ in range(5):
            ops += [W.Op(ry(rng.uniform(0, 6)), [q]) for q in range(n)]
            ops += [W.Op(W.X.copy(), [t], {c}) for c, t in pairs]
        check(lib, n, ops, 8950 + seed)

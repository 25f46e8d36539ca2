"""Merged one-qubit gates in the factored-sweep planner (doki_b200/csrc/dk_plan_fx.c),
on CPU: gates are multiplied into the next gate on their qubit, and roundings of
the matrices add up along a run until a product no longer factors.  Every gate has
to be in the plan all the same, and a plan whose gates all factor has to consist of
factored programs only: its readers take them for nothing else."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.test_plan import HDR, lib  # noqa: F401
from tests.test_plan_factored import plan, run


def rounded(m, digits):
    return np.round(m.real, digits) + 1j * np.round(m.imag, digits)


def product(rng, count):
    m = np.eye(2, dtype=np.complex128)
    for _ in range(count):
        m = W.u3(*rng.uniform(0, 6, 3)) @ m
    return m


def long_apply(psi, op):
    """One gate on a state in extended precision."""
    t = op.targets[0]
    idx = np.arange(psi.size)
    on = np.ones(psi.size, dtype=bool)
    for c in op.controls:
        on &= (idx >> c) & 1 == 1
    m = np.asarray(op.gate).astype(np.clongdouble)
    i0 = idx[on & ((idx >> t) & 1 == 0)]
    i1 = i0 | (1 << t)
    a, b = psi[i0].copy(), psi[i1].copy()
    psi[i0], psi[i1] = m[0, 0] * a + m[0, 1] * b, m[1, 0] * a + m[1, 1] * b


def check(lib, n, ops, tol=2e-12):  # noqa: F811
    rng = W.rng_for(n)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    want = psi.astype(np.clongdouble)
    for op in ops:
        long_apply(want, op)
    got, kinds = run(lib, ops, n, psi)  # also: the steps' gates add up to len(ops)
    assert set(kinds) == {2}
    err = np.max(np.abs(got - want.astype(np.complex128))) / np.max(np.abs(want))
    assert err < tol, float(err)


# Tolerance: a merged run of gates drops at most 1e-13 of its product where it ends,
# one run per 100 gates or more; in between the roundings are those of extended
# precision.  2000 gates: 20 runs.

@pytest.mark.parametrize("repeats", [300, 1000, 2000])
def test_one_gate_many_times(lib, repeats):  # noqa: F811
    """Some of these angles give matrices whose 300th, 1000th or 2000th power no
    longer factors."""
    for seed in range(24):
        u = W.u3(*np.random.default_rng(seed).uniform(0, 6, 3))
        check(lib, 6, [W.Op(u, [0])] * repeats)


@pytest.mark.parametrize("kind", ["products", "14 digits"])
def test_matrices_that_are_a_little_off(lib, kind):  # noqa: F811
    """Products of 60 matrices, and matrices written down with 14 digits, each
    repeated up to 200 times: their runs end after a few gates."""
    for seed in range(12):
        rng = W.rng_for(8100 + seed)
        m = product(rng, 60) if kind == "products" else rounded(W.u3(*rng.uniform(0, 6, 3)), 14)
        for repeats in (20, 50, 200):
            ops = [W.Op(m, [1])] * repeats
            rngs = np.random.default_rng(seed)
            psi = rngs.normal(size=64) + 1j * rngs.normal(size=64)
            want = psi.astype(np.clongdouble)
            for op in ops:
                long_apply(want, op)
            got, _ = run(lib, ops, 6, psi)
            err = np.max(np.abs(got - want.astype(np.complex128))) / np.max(np.abs(want))
            assert err < 2e-12, (seed, repeats, float(err))


def test_factors_through_controls_and_x(lib):  # noqa: F811
    """Long runs whose factors also move through X, CNOTs and diagonal gates: a
    phase or a rotation that no later gate can take stays where it was."""
    for seed in range(10):
        rng = W.rng_for(8200 + seed)
        base = [W.u3(*rng.uniform(0, 6, 3)) for _ in range(3)]
        ops = []
        for i in range(900):
            q = int(rng.integers(0, 3))
            r = rng.random()
            if r < 0.8:
                ops.append(W.Op(base[q], [q]))
            elif r < 0.88:
                ops.append(W.Op(W.X.copy(), [q], {(q + 1) % 3}))
            elif r < 0.94:
                ops.append(W.Op(W.X.copy(), [q]))
            elif r < 0.97:
                ops.append(W.Op(np.diag([1, np.exp(1j * rng.random())]), [q], {(q + 1) % 3}))
            else:
                ops.append(W.Op(np.diag(np.exp(1j * rng.random(2))), [q]))
        check(lib, 6, ops)


@pytest.mark.parametrize("prec", [2, 1])
def test_plans_that_factor_hold_factored_programs_only(lib, prec):  # noqa: F811
    """What dk_fx_all promises."""
    for seed in range(40):
        rng = W.rng_for(8300 + seed)
        u = W.u3(*rng.uniform(0, 6, 3))
        if seed % 2:
            u = rounded(u, 14)
        ops = [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q]) for q in range(6)] + [W.Op(u, [2])] * 1000
        for m in {tuple(op.gate.reshape(-1)) for op in ops}:
            one = plan(lib, [W.Op(np.array(m).reshape(2, 2), [0])], 6, prec)
            if np.frombuffer(one[0][1], HDR, 1)[0]["mode"] != 2:
                break  # a matrix that does not factor by itself
        else:
            steps = plan(lib, ops, 6, prec)
            assert all(k == 1 and np.frombuffer(b, HDR, 1)[0]["mode"] == 2 for k, b, _, _ in steps)
            assert sum(s[3] for s in steps) == len(ops)

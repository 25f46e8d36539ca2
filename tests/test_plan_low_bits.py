"""The low qubits that a sweep's tile always holds, on CPU: a wider run for factored
sweeps leaves the sweeps of dense gates as they are without it."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.golden.gen_golden import random_unitary
from tests.test_plan import HDR, FlatOp, Limits, Step, build_plan, lib  # noqa: F401


def sweeps(lib, ops, n, prec, low):  # noqa: F811
    """(mode, tile qubits) of the streamed plan's sweeps; -1: a generic gate."""
    lib.dk_fx_begin.argtypes = [ctypes.POINTER(FlatOp), ctypes.c_int, ctypes.c_uint, ctypes.c_int,
                                ctypes.POINTER(Limits), ctypes.POINTER(ctypes.c_void_p)]
    lib.dk_fx_next.argtypes = [ctypes.c_void_p, ctypes.POINTER(Step),
                               ctypes.POINTER(ctypes.c_void_p)]
    lib.dk_fx_set_low_bits.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.dk_fx_end.argtypes = [ctypes.c_void_p]
    flat, gates, out = (FlatOp * len(ops))(), [], []
    for i, op in enumerate(ops):
        m = np.ascontiguousarray(op.gate, dtype=np.complex128)
        g = ctypes.c_void_p()
        assert lib.dk_gate_new(op.k, m.ctypes.data, ctypes.byref(g)) == 0
        gates.append(g)
        flat[i].gate, flat[i].k = g, op.k
        for j, t in enumerate(op.targets):
            flat[i].tg[j] = t
        flat[i].cm = sum(1 << c for c in op.controls)
        flat[i].am = sum(1 << c for c in op.anticontrols)
    lim, h = Limits(), ctypes.c_void_p()
    lib.dk_plan_default_limits(prec, n, ctypes.byref(lim))
    lim.bank_mode = 1 if prec == 1 else 0
    assert lib.dk_fx_begin(flat, len(ops), n, prec, ctypes.byref(lim), ctypes.byref(h)) == 0
    if low is not None:
        lib.dk_fx_set_low_bits(h, low)
    gates_done = 0
    while True:
        step, prog = Step(), ctypes.c_void_p()
        rc = lib.dk_fx_next(h, ctypes.byref(step), ctypes.byref(prog))
        assert rc in (0, 1)
        if rc == 0:
            break
        gates_done += step.ngates
        if step.kind != 1:
            out.append((-1, ()))
            continue
        hdr = np.frombuffer(ctypes.string_at(prog.value, HDR.itemsize), HDR, 1)[0]
        out.append((int(hdr["mode"]), tuple(int(q) for q in hdr["qpos"][:int(hdr["m"])])))
    assert gates_done == len(ops)
    lib.dk_fx_end(h)
    for g in gates:
        lib.dk_gate_free(g)
    return out


def brickwork(n, depth, seed):
    rng = W.rng_for(seed)
    return [W.Op(random_unitary(rng, 2), [a, a + 1])
            for layer in range(depth) for a in range(layer % 2, n - 1, 2)]


@pytest.mark.parametrize("n,want", [(24, 21), (28, 25)])
def test_dense_sweeps_keep_their_number(lib, n, want):  # noqa: F811
    ops = brickwork(n, 20, n)
    steps, _ = build_plan(lib, ops, n, 1, bank_mode=1)
    assert len(steps) == want
    got = sweeps(lib, ops, n, 1, 4)
    assert {m for m, _ in got} == {1} and len(got) == want


def test_each_kind_has_its_own_run(lib):  # noqa: F811
    """Factored sweeps hold the 4 low qubits, dense ones only those they need."""
    n = 26
    ops = W.scale_circuit(seed=1, n=n, depth=4).ops + brickwork(n, 6, 1)
    ops += W.scale_circuit(seed=2, n=n, depth=4).ops
    got = sweeps(lib, ops, n, 1, 4)
    assert {m for m, _ in got} == {1, 2}
    assert all(set(range(4)) <= set(q) for m, q in got if m == 2)
    assert all(set(range(2)) <= set(q) for _, q in got)
    assert any(not set(range(4)) <= set(q) for m, q in got if m == 1)
    # without a choice of its own a factored sweep takes the limits' run
    assert any(not set(range(4)) <= set(q) for m, q in sweeps(lib, ops, n, 1, None) if m == 2)

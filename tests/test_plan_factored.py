"""Host logic of the factored-sweep planner (doki_b200/csrc/dk_plan_fx.c), on
CPU: its programs, read back through ctypes and replayed by a numpy model of
the kernel (gather, operation list of the tile's conditions, scatter, by shared
memory slot), must equal gate-by-gate application by the oracle."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.golden.gen_golden import random_unitary
from tests.test_plan import (COND, HDR, FlatOp, Limits, Step, apply_local, lib,  # noqa: F401
                             oracle_run, random_ops, replay_sweep, swizzle_map)

PASS = np.dtype([("flags", "<u4"), ("list", "<u4"), ("cond", "<u4"), ("pad", "<u4"),
                 ("pm", "<u2", 4), ("shi", "<u2", 8), ("slo", "<u2", 32), ("rhi", "<u2", 8),
                 ("rlo", "<u2", 32), ("pad2", "<u2", 4)])
LIST = np.dtype([("gt", "<u2", 4), ("st", "<u2", 4), ("gc", "<u2"), ("sc", "<u2"),
                 ("op0", "<u2"), ("op1", "<u2"), ("lmap", "<u4"), ("idle", "<u4")])
OP = np.dtype([("code", "<u2"), ("mask", "<u2"), ("coef", "<u4"), ("lc", "<u4"), ("la", "<u4")])
assert PASS.itemsize == 192 and LIST.itemsize == 32 and OP.itemsize == 16


def plan(lib, ops, n, prec=2, tile_bits=None):  # noqa: F811
    """[(kind, program bytes or None, op index)] of the streamed plan."""
    lib.dk_fx_begin.argtypes = [ctypes.POINTER(FlatOp), ctypes.c_int, ctypes.c_uint, ctypes.c_int,
                                ctypes.POINTER(Limits), ctypes.POINTER(ctypes.c_void_p)]
    lib.dk_fx_next.argtypes = [ctypes.c_void_p, ctypes.POINTER(Step),
                               ctypes.POINTER(ctypes.c_void_p)]
    lib.dk_fx_end.argtypes = [ctypes.c_void_p]
    flat, gates = (FlatOp * len(ops))(), []
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
    lim = Limits()
    lib.dk_plan_default_limits(prec, n, ctypes.byref(lim))
    if tile_bits is not None:
        lim.tile_bits = tile_bits
    h, out = ctypes.c_void_p(), []
    assert lib.dk_fx_begin(flat, len(ops), n, prec, ctypes.byref(lim), ctypes.byref(h)) == 0
    while True:
        step, prog = Step(), ctypes.c_void_p()
        rc = lib.dk_fx_next(h, ctypes.byref(step), ctypes.byref(prog))
        assert rc in (0, 1), rc
        if rc == 0:
            break
        blob = None
        if step.kind == 1:
            hdr = np.frombuffer(ctypes.string_at(prog.value, HDR.itemsize), HDR, 1)[0]
            blob = ctypes.string_at(prog.value, int(hdr["bytes"]))
        out.append((step.kind, blob, step.op_index, step.ngates))
    lib.dk_fx_end(h)
    for g in gates:
        lib.dk_gate_free(g)
    return out


def reals(coef, at, cnt, prec):
    """The (x, y) of the 8 pairs of a rotation (one for all when cnt = 1)."""
    if prec == 2:
        co = np.frombuffer(coef, "<f8", 2 * cnt, at).reshape(cnt, 2)
    else:
        co = np.frombuffer(coef, "<f4", 4 * cnt, at).reshape(cnt, 4)
        assert np.array_equal(co[:, 0], co[:, 1]) and np.array_equal(co[:, 2], co[:, 3])
        co = co[:, ::2]
    return np.broadcast_to(co.astype(np.float64), (8, 2))


def rotate(a, ok, d, co):
    pairs = [(x, x ^ d) for x in range(16) if not x & (d & -d)]
    for (x, y), (cx, cy) in zip(pairs, co):
        ax, ay = a[ok, x].copy(), a[ok, y].copy()
        a[ok, x], a[ok, y] = ax + cx * ay, ay + cy * ax


def replay(blob, psi, prec):
    """One factored program on a state; checks the tables on the way."""
    h = np.frombuffer(blob, HDR, 1)[0]
    m, n = int(h["m"]), int(h["n"])
    assert int(h["mode"]) == 2
    passes = np.frombuffer(blob, PASS, int(h["npass"]), int(h["pass_off"]))
    amp = 16 if prec == 2 else 8
    nlist = max(int(p["list"]) + (1 << (int(p["cond"]) >> 15)) for p in passes)
    list_off = int(h["pass_off"]) + PASS.itemsize * int(h["npass"])
    assert list_off + LIST.itemsize * nlist == int(h["gate_off"]) and int(h["ncond"]) <= 32
    lists = np.frombuffer(blob, LIST, nlist, list_off)
    ops = np.frombuffer(blob, OP, int(h["ngate"]), int(h["gate_off"]))
    conds = np.frombuffer(blob, COND, int(h["ncond"]), int(h["cond_off"]))
    coef = blob[int(h["mat_off"]):int(h["bytes"])]
    qpos = [int(q) for q in h["qpos"][:m]]
    local = np.arange(1 << m)
    offs = np.zeros(1 << m, dtype=np.int64)
    for j, q in enumerate(qpos):
        offs |= ((local >> j) & 1) << q
    slot_of = np.array([swizzle_map(int(i), h["bankv"]) for i in local])
    assert sorted(slot_of) == list(local)
    rest = [q for q in range(n) if q not in qpos]
    nt = 1 << (m - 4)
    tid, reg = np.arange(nt), np.arange(16)

    def lin(vec):  # XOR of vec[j] over the bits of the register number
        return np.bitwise_xor.reduce([np.where((reg >> j) & 1, int(vec[j]), 0) for j in range(4)])

    out = psi.copy()
    for t in range(int(h["ntiles"])):
        base = sum(((t >> j) & 1) << q for j, q in enumerate(rest))
        tile = np.empty(1 << m, dtype=np.complex128)
        tile[slot_of] = out[base | offs]
        if not int(h["all_touched"]):
            assert len(conds) > 0
        for p in passes:
            v = 0
            for c in range(int(p["cond"]) >> 15):
                gc, ga = (int(x) for x in conds[(int(p["cond"]) >> (5 * c)) & 31])
                v |= ((base & gc) == gc and not base & ga) << c
            li = lists[int(p["list"]) + v]
            raw = p["rlo"][tid & 31].astype(np.int64) | p["rhi"][tid >> 5]
            sg = (p["slo"][tid & 31].astype(np.int64) ^ p["shi"][tid >> 5]) // amp
            full = raw[:, None] | lin(p["pm"])[None, :]
            assert sorted(full.ravel()) == list(local)
            assert np.array_equal(sg, slot_of[raw])
            slots = sg[:, None] ^ lin(li["gt"] // amp)[None, :] ^ int(li["gc"]) // amp
            assert np.array_equal(np.sort(slots, 1), np.sort(slot_of[full], 1))
            a = tile[slots]
            for o in ops[int(li["op0"]):int(li["op1"])]:
                lc, la = int(o["lc"]), int(o["la"])
                assert not (lc | la) or int(p["flags"]) & 1
                ok = ((raw & lc) == lc) & ((raw & la) == 0)
                code, at, mask = int(o["code"]), 16 * int(o["coef"]), int(o["mask"])
                dt = "<c16" if prec == 2 else "<c8"
                inm = (mask >> reg) & 1 == 1
                if code == 0:
                    if mask & 16:
                        a[ok] = a[ok] * np.frombuffer(coef, dt, 16, at + 64)
                    for j in range(4):
                        if (mask >> j) & 1:
                            rotate(a, ok, 1 << j, reals(coef, at + 16 * j, 1, prec))
                    continue
                if code in (16, 32):
                    u = np.frombuffer(coef, dt, 1, at)[0] if code == 16 else -1
                    a[np.ix_(ok, inm)] *= u
                    continue
                d = code & 15
                pairs = [(x, x ^ d) for x in range(16) if not x & (d & -d)]
                if 16 < code < 32:
                    for i, (x, y) in enumerate(pairs):
                        if (mask >> i) & 1:
                            a[np.ix_(ok, [x, y])] = a[np.ix_(ok, [y, x])]
                    continue
                rotate(a, ok, d, reals(coef, at, 8, prec))
            sl = sg[:, None] ^ lin(li["st"] // amp)[None, :] ^ int(li["sc"]) // amp
            assert sorted(sl.ravel()) == list(local)
            if int(li["idle"]):
                assert np.array_equal(sl, slots) and li["op0"] == li["op1"]
            # the same map as pass indices, for a pass that stores to the register
            lm = int(li["lmap"])
            lab = np.bitwise_xor.reduce([np.where((reg >> j) & 1, (lm >> (4 * j)) & 15, 0)
                                         for j in range(4)]) ^ (lm >> 16)
            bits = sum(((lab >> j) & 1) * int(p["pm"][j]) for j in range(4))
            assert np.array_equal(sl, slot_of[raw[:, None] | bits[None, :]])
            if int(p["flags"]) & 4:
                assert p is passes[-1] or p["flags"] == passes[-1]["flags"]
                lane_bits = sum(int(p["rlo"][1 << j]) for j in range(min(5, m - 4)))
                assert lane_bits & 3 == 3
            tile[sl] = a
        out[base | offs] = tile[slot_of]
    return out


def run(lib, ops, n, psi, prec=2, tile_bits=None):  # noqa: F811
    steps = plan(lib, ops, n, prec, tile_bits)
    kinds = []
    for kind, blob, opi, _ in steps:
        if kind == 1:
            mode = int(np.frombuffer(blob, HDR, 1)[0]["mode"])
            kinds.append(mode)
            psi = replay(blob, psi, prec) if mode == 2 else replay_sweep(blob, 0, psi)
        else:
            kinds.append(-1)
            op = ops[opi]
            idx = np.arange(psi.size)
            cm = sum(1 << c for c in op.controls)
            am = sum(1 << c for c in op.anticontrols)
            psi = apply_local(psi, op.gate, list(op.targets),
                              ((idx & cm) == cm) & ((idx & am) == 0))
    assert sum(s[3] for s in steps) == len(ops)
    return psi, kinds


def one_qubit_ops(rng, n, count):
    """Gates that all have a factoring: U3, H, X, Y, Z, S, phases, Ry near pi,
    anti-diagonal matrices, real non-unitary ones, 2- and 3-qubit diagonals, with
    up to three controls and anticontrols anywhere."""
    out = []
    for _ in range(count):
        k, r = 1, rng.random()
        ph = np.exp(2j * np.pi * rng.random(8))
        if r < 0.45:
            m = W.u3(*rng.uniform(0, 2 * np.pi, 3))
        elif r < 0.6:
            m = [W.H, W.X, W.Z, np.array([[0, -1j], [1j, 0]])][int(rng.integers(4))]
        elif r < 0.7:
            m = W.u3(np.pi * (1 + [0, 1e-3, -1e-9][int(rng.integers(3))]), *rng.uniform(0, 6, 2))
        elif r < 0.75:
            m = np.diag([1, ph[0]])
        elif r < 0.8:
            m = np.diag(ph[:2])
        elif r < 0.85:
            m = np.array([[0, ph[0]], [ph[1], 0]])
        elif r < 0.9:
            m = np.array([[1.0, 0.5], [-0.25, 1.5]])
        else:
            k = 2 + int(rng.integers(2))
            m = np.diag(ph[:1 << k])
        q = [int(x) for x in rng.permutation(n)]
        nc = min(n - k, int(rng.integers(0, 4))) if rng.random() < 0.6 else 0
        cs = q[k:k + nc]
        ctl = {c for c in cs if rng.random() < 0.6}
        out.append(W.Op(np.asarray(m, dtype=np.complex128), q[:k], ctl, set(cs) - ctl))
    return out


@pytest.mark.parametrize("n,tile_bits", [(4, None), (5, None), (6, None), (8, None), (10, 6),
                                         (9, None), (10, None), (12, None), (12, 9), (13, 10),
                                         (14, None), (14, 11)])
def test_factored_replay_matches_oracle(lib, orc, n, tile_bits):  # noqa: F811
    rng = W.rng_for(7000 + n + (tile_bits or 0))
    ops = one_qubit_ops(rng, n, 90) + W.scale_circuit(seed=n, n=n, depth=3, ctrl_frac=0.3).ops
    psi0 = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    got, kinds = run(lib, ops, n, psi0, tile_bits=tile_bits)
    assert set(kinds) == {2}
    reg = W.run_ops(orc, orc.registry_new_data(n, psi0), ops)
    want = orc.registry_get_all(reg)
    assert np.allclose(got / np.linalg.norm(got), want, atol=1e-12)


@pytest.mark.parametrize("n,tile_bits", [(1, None), (2, None), (3, None), (5, 3)])
def test_small_tiles_take_the_other_planner(lib, orc, n, tile_bits):  # noqa: F811
    """Registers and tiles below 4 qubits: no factored sweep, and no gate merged
    into another."""
    rng = W.rng_for(7100 + n)
    ops = []
    for _ in range(30):
        q = [int(x) for x in rng.permutation(n)]
        ops.append(W.Op(W.u3(*rng.uniform(0, 6, 3)), q[:1], set(q[1:1 + int(rng.integers(0, 2))])))
    psi0 = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    got, kinds = run(lib, ops, n, psi0, tile_bits=tile_bits)
    assert 2 not in kinds
    want = orc.registry_get_all(W.run_ops(orc, orc.registry_new_data(n, psi0), ops))
    assert np.allclose(got / np.linalg.norm(got), want, atol=1e-12)


def test_factored_complex64_programs(lib, orc):  # noqa: F811
    """The single-precision tables: 16 roundings of 2^-24 per gate and
    amplitude at most, 150 gates, amplitudes below 0.1: within 1e-4, and
    typically 1e-7."""
    n = 13
    rng = W.rng_for(77)
    ops = one_qubit_ops(rng, n, 60) + W.small_circuit(seed=3, n=n, depth=4).ops
    psi0 = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi0 /= np.linalg.norm(psi0)
    got, kinds = run(lib, ops, n, psi0, prec=1)
    assert set(kinds) == {2}
    want = orc.registry_get_all(W.run_ops(orc, orc.registry_new_data(n, psi0), ops))
    assert np.max(np.abs(got / np.linalg.norm(got) - want)) < 2e-6


def test_gates_without_a_factoring_take_the_other_planner(lib, orc):  # noqa: F811
    """Dense 2- and 3-qubit gates, a one-qubit matrix whose b c / (a d) is not
    real and a 4-qubit gate, among gates that factor."""
    n = 13
    rng = W.rng_for(78)
    skew = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
    ops = random_ops(rng, n, 50) + [W.Op(skew, [3], {1}), W.Op(random_unitary(rng, 4), [0, 12, 5, 2])]
    ops += one_qubit_ops(rng, n, 50)
    psi0 = np.zeros(1 << n, dtype=np.complex128)
    psi0[0] = 1
    got, kinds = run(lib, ops, n, psi0)
    assert {-1, 1, 2} <= set(kinds)
    want = oracle_run(orc, ops, n)
    assert np.allclose(got / np.linalg.norm(got), want / np.linalg.norm(want), atol=1e-12)


def test_permutations_and_phases_keep_zeros_exact(lib):  # noqa: F811
    """X, CNOT, Toffoli and diagonal gates only move and scale amplitudes: a
    basis state stays one, every other amplitude exactly 0."""
    n = 14
    rng = W.rng_for(79)
    ops = []
    for _ in range(80):
        q = [int(x) for x in rng.permutation(n)]
        nc = int(rng.integers(0, 3))
        g = [W.X, W.Z, np.diag([1, 1j])][int(rng.integers(3))]
        ops.append(W.Op(g.astype(np.complex128), [q[0]], set(q[1:1 + nc])))
    psi0 = np.zeros(1 << n, dtype=np.complex128)
    psi0[5] = 1
    got, kinds = run(lib, ops, n, psi0)
    assert set(kinds) == {2}
    assert np.count_nonzero(got) == 1 and np.max(np.abs(got)) == 1.0


def test_long_programs_are_cut(lib, orc):  # noqa: F811
    """Hundreds of gates on the same few qubits with three tile conditions:
    programs stay within their bound and the gates keep their order."""
    n = 20
    rng = W.rng_for(80)
    ops = []
    for i in range(150):
        q = int(rng.integers(0, 4))
        far = {int(19 - rng.integers(0, 3))} if rng.random() < 0.5 else set()
        ops.append(W.Op(W.u3(*rng.uniform(0, 6, 3)), [q], far))
    steps = plan(lib, ops, n)
    assert len(steps) > 1 and sum(s[3] for s in steps) == len(ops)
    assert all(len(s[1]) <= 40 << 10 for s in steps)
    psi0 = np.zeros(1 << n, dtype=np.complex128)
    psi0[rng.integers(0, 1 << n, 64)] = rng.normal(size=64)
    got, _ = run(lib, ops, n, psi0)
    want = orc.registry_get_all(W.run_ops(orc, orc.registry_new_data(n, psi0), ops))
    assert np.allclose(got / np.linalg.norm(got), want, atol=1e-12)

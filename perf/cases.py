"""Timed cases: the work a program has this engine do, through its public calls.

Every case is one of six kinds of use of the `doki` module and the batch
engine (``doki_b200``):

- ``circuit``: a whole circuit on a fresh register and its results
  (probabilities, measurement with the register that is left, reduced density
  matrix), queued gate by gate (``registry_apply``, as programs written for
  the original module do) or as one prepared circuit (``registry_apply_many``,
  the serving form);
- ``steps``: gates applied one at a time with a probability read after each
  (interactive and adaptive programs: nothing can be fused across a read);
- ``measure``: a register in hand, some of its qubits measured;
- ``density``: a register in hand, its reduced density matrix;
- ``join``: two registers in hand, their product and its probabilities;
- ``batch``: many small circuits planned once and run as one batch.

Sizes are those of this repository's workloads (the 12-qubit depth-20 circuit,
the 30-qubit depth-40 job, requests of 8 to 28 qubits and depth 10 to 100,
batches of 4 to 16 qubits and depth 10 to 50) and odd ones between.  Values
read from a complex64 register carry single precision and are kept as such.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import doki_b200
from doki_b200 import workloads as W
from doki_b200.batch import BatchEngine


def listed():
    return [
        # the smallest calls: a first circuit of a few gates, every result read
        {"name": "first_circuit_6q", "kind": "circuit", "family": "layers", "n": 6, "depth": 2,
         "precision": 2, "entry": "gates", "measure": 0, "keep": 0, "amps": True},
        # the 12-qubit depth-20 circuit, gate by gate, all qubits measured
        {"name": "circuit_12q", "kind": "circuit", "family": "layers", "n": 12, "depth": 20,
         "precision": 2, "entry": "gates", "measure": 12, "keep": 0, "amps": True},
        # serving requests: small, middle, and the largest a stream holds
        {"name": "request_17q_c64", "kind": "circuit", "family": "layers", "n": 17, "depth": 37,
         "precision": 1, "entry": "many", "measure": 0, "keep": 0, "amps": True},
        {"name": "request_23q_c64", "kind": "circuit", "family": "layers", "n": 23, "depth": 61,
         "precision": 1, "entry": "many", "measure": 5, "keep": 0, "amps": False},
        {"name": "request_28q_c64", "kind": "circuit", "family": "layers", "n": 28, "depth": 55,
         "precision": 1, "entry": "many", "measure": 8, "keep": 0, "amps": False},
        # a brickwork circuit whose register stays in the L2 cache
        {"name": "brick_21q", "kind": "circuit", "family": "brick", "n": 21, "depth": 33,
         "precision": 2, "entry": "many", "measure": 3, "keep": 7, "amps": False},
        # the 30-qubit job: depth 40, all marginals, 4 measured, 10 kept
        {"name": "scale_30q", "kind": "circuit", "family": "brick", "n": 30, "depth": 40,
         "precision": 2, "entry": "many", "measure": 4, "keep": 10, "amps": False},
        # a program that reads a probability after every gate
        {"name": "steps_24q", "kind": "steps", "n": 24, "gates": 9, "precision": 2},
        # mid-circuit measurement of scattered qubits of a register in hand
        {"name": "measure_27q", "kind": "measure", "n": 27, "measure": 7, "precision": 2},
        # reduced density matrix over scattered qubits
        {"name": "density_25q_c64", "kind": "density", "n": 25, "keep": 9, "low": False,
         "precision": 1},
        # a product register
        {"name": "join_26q", "kind": "join", "most": 11, "least": 15, "precision": 2},
        # many small circuits at once
        {"name": "batch_1024_c64", "kind": "batch", "count": 1024, "qmin": 4, "qmax": 16,
         "dmin": 10, "dmax": 50, "precision": 1, "tile_bits": 12, "ctas": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "steps", "measure", "density", "join",
                       "batch"])
    prec = rng.choice([1, 2])
    if kind == "circuit":
        # amplitudes are spread over their logarithm: qubits uniformly
        n = rng.randint(4, 28)
        depth = _log_int(rng, 2, 100 if n <= 24 else 40)
        entry = rng.choice(["gates", "many"])
        return {"kind": kind, "family": rng.choice(["layers", "brick"]), "n": n, "depth": depth,
                "precision": prec, "entry": entry, "measure": rng.randint(0, min(n, 14)),
                "keep": rng.choice([0, rng.randint(1, min(n, 9))]), "amps": n <= 19}
    if kind == "steps":
        return {"kind": kind, "n": rng.randint(5, 27), "gates": rng.randint(2, 16),
                "precision": prec}
    if kind == "measure":
        n = rng.randint(6, 28)
        return {"kind": kind, "n": n, "measure": rng.randint(1, min(n - 1, 14)),
                "precision": prec}
    if kind == "density":
        n = rng.randint(8, 26)
        return {"kind": kind, "n": n, "keep": rng.randint(1, min(n, 10)),
                "low": rng.random() < 0.5, "precision": prec}
    if kind == "join":
        n = rng.randint(6, 28)
        most = rng.randint(1, n - 1)
        return {"kind": kind, "most": most, "least": n - most, "precision": prec}
    qmin = rng.randint(4, 10)
    return {"kind": kind, "count": _log_int(rng, 16, 1024), "qmin": qmin,
            "qmax": rng.randint(qmin, 16), "dmin": 10, "dmax": rng.randint(10, 50),
            "precision": prec, "tile_bits": rng.choice([11, 12]), "ctas": rng.choice([1, 2])}


# ---- circuits as data -----------------------------------------------------

def _rng(case, seed):
    return np.random.default_rng([int(seed), 1009 * int(case.get("n", 0)) + 7])


def _ops(case, seed):
    s = int(seed) % (1 << 31)
    if case["family"] == "layers":
        return W.small_circuit(seed=s, n=case["n"], depth=case["depth"]).ops
    return W.scale_circuit(seed=s, n=case["n"], depth=case["depth"],
                           n_measure=1, keep=1).ops


def _flat(ops):
    """Gates as the arrays of registry_apply_many."""
    k = np.array([op.k for op in ops], dtype=np.uint32)
    tg = np.zeros((len(ops), 3), dtype=np.uint32)
    cm = np.zeros(len(ops), dtype=np.uint64)
    am = np.zeros(len(ops), dtype=np.uint64)
    mi = np.zeros(len(ops), dtype=np.uint64)
    mats, off = [], 0
    for i, op in enumerate(ops):
        tg[i, :op.k] = op.targets
        cm[i] = sum(1 << q for q in op.controls)
        am[i] = sum(1 << q for q in op.anticontrols)
        mi[i] = off
        mats.append(np.ascontiguousarray(op.gate, dtype=np.complex128).reshape(-1))
        off += mats[-1].size
    return k, tg, cm, am, mi, np.concatenate(mats)


def _ending(case, seed, n):
    """Measured qubits with their rolls, and the kept qubits."""
    rng = np.random.default_rng([int(seed), 77, n])
    perm = [int(q) for q in rng.permutation(n)]
    mask = sum(1 << q for q in perm[:case.get("measure", 0)])
    rolls = rng.random(case.get("measure", 0)).tolist()
    k = case.get("keep", 0)
    if case["kind"] == "density" and not case["low"]:
        keep = sorted(perm[:k])
    else:
        keep = list(range(k))
    return mask, rolls, keep


def _random_layer(rng, n):
    """One-qubit gates on every qubit and a chain of entangling ones: a cheap
    way to a register whose amplitudes are all different."""
    ops = [W.Op(W.u3(*(rng.random(3) * 2 * np.pi)), [q]) for q in range(n)]
    ops += [W.Op(W.X.copy(), [q + 1], {q}) for q in range(n - 1)]
    ops += [W.Op(W.u3(*(rng.random(3) * 2 * np.pi)), [q]) for q in range(n)]
    return ops


def _step_ops(case, seed):
    rng = _rng(case, seed)
    n = case["n"]
    ops = []
    for i in range(case["gates"]):
        q, c = (int(x) for x in rng.choice(n, size=2, replace=False))
        if i % 3 == 2:
            ops.append(W.Op(W.X.copy(), [q], {c}))
        else:
            ops.append(W.Op(W.u3(*(rng.random(3) * 2 * np.pi)), [q]))
    return ops


def _batch(case, seed):
    """Widths, depths and pairings follow from the case, angles from the seed."""
    flat = W.batch_arrays(seed=case["count"], count=case["count"], qmin=case["qmin"],
                          qmax=case["qmax"], dmin=case["dmin"], dmax=case["dmax"])
    rng = np.random.default_rng([int(seed), case["count"]])
    th, ph, la = rng.random((3, flat.matrices.size // 4 - 1)) * 2 * np.pi
    c, s = np.cos(th / 2), np.sin(th / 2)
    u = np.stack([c, -np.exp(1j * la) * s, np.exp(1j * ph) * s, np.exp(1j * (ph + la)) * c], 1)
    flat.matrices[4:] = u.reshape(-1)  # the first matrix is X
    return flat


def _register(d, ops, n, precision):
    reg = d.registry_apply_many(d.registry_new(n, False, precision), *_flat(ops))
    d.registry_flush(reg)
    return reg


def _gate_calls(d, ops):
    calls = []
    for op in ops:
        ctl = set(op.controls) if (op.controls or op.anticontrols) else None
        calls.append((d.gate_new(op.k, op.gate.tolist(), False), list(op.targets), ctl,
                      set(op.anticontrols) or None))
    return calls


# ---- the measured pass ------------------------------------------------------

def prepare(case, seed):
    d = doki_b200.load()
    kind = case["kind"]
    s = {"d": d, "case": case, "kind": kind}
    if kind == "batch":
        s["engine"] = BatchEngine(_batch(case, seed), case["precision"], tile_bits=case["tile_bits"],
                                  ctas_per_sm=case["ctas"])
        s["out"] = torch.empty(s["engine"].rho_elems, dtype=torch.complex128,
                               pin_memory=torch.cuda.is_available())
        if case["precision"] == 1:
            s["single"] = torch.empty(s["engine"].rho_elems, dtype=torch.complex64)
        return s
    if kind == "join":
        rng = _rng(case, seed)
        s["most"] = _register(d, _random_layer(rng, case["most"]), case["most"],
                              case["precision"])
        s["least"] = _register(d, _random_layer(rng, case["least"]), case["least"],
                               case["precision"])
        return s
    n = case["n"]
    s["mask"], s["rolls"], s["keep"] = _ending(case, seed, n)
    if kind == "circuit":
        ops = _ops(case, seed)
        if case["entry"] == "gates":
            s["calls"] = _gate_calls(d, ops)
        else:
            s["arrays"] = _flat(ops)
        return s
    s["reg"] = _register(d, _random_layer(_rng(case, seed), n), n, case["precision"])
    if kind == "steps":
        s["calls"] = _gate_calls(d, _step_ops(case, seed))
    return s


def _real(case, values):
    return np.asarray(values, dtype=np.float64 if case["precision"] == 2 else np.float32)


def _complex(case, values):
    return np.asarray(values, dtype=np.complex128 if case["precision"] == 2 else np.complex64)


def _measured(s, reg):
    """Outcomes and the probabilities of the register that is left."""
    d = s["d"]
    left, res = d.registry_measure(reg, s["mask"], s["rolls"], -1, False)
    out = {"outcomes": np.array([-1 if r is None else int(r) for r in res], dtype=np.int64)}
    if left is not None:
        out["left"] = _real(s["case"], d.registry_probs(left))
    return out


def _density(s, reg, n):
    d = s["d"]
    rho = d.registry_density(reg, False)
    for q in range(n - 1, -1, -1):
        if q not in s["keep"]:
            rho = d.funmatrix_partialtrace(rho, q, False)
    return _complex(s["case"], d.funmatrix_numpy(rho))


def run(state):
    s = state
    d, case, kind = s["d"], s["case"], s["kind"]
    if kind == "batch":
        s["engine"].run()
        s["engine"].rho_all(s["out"].numpy())
        return s["single"].copy_(s["out"]) if case["precision"] == 1 else s["out"]
    if kind == "join":
        reg = d.registry_join(s["most"], s["least"], -1, False)
        return _real(case, d.registry_probs(reg))
    n = case["n"]
    if kind == "measure":
        return _measured(s, s["reg"])
    if kind == "density":
        return _density(s, s["reg"], n)
    if kind == "steps":
        reg, probs = s["reg"], []
        for gate, targets, ctl, actl in s["calls"]:
            reg = d.registry_apply(reg, gate, targets, ctl, actl, -1, False)
            probs.append(d.registry_prob(reg, targets[0], -1, False))
        return {"after_each": _real(case, probs), "probs": _real(case, d.registry_probs(reg))}
    reg = d.registry_new(n, False, case["precision"])
    if case["entry"] == "gates":
        for gate, targets, ctl, actl in s["calls"]:
            reg = d.registry_apply(reg, gate, targets, ctl, actl, -1, False)
    else:
        reg = d.registry_apply_many(reg, *s["arrays"])
    out = {"probs": _real(case, d.registry_probs(reg))}
    if case["amps"]:
        out["amps"] = _complex(case, d.registry_get_all(reg, False))
    if case["keep"]:
        out["rho"] = _density(s, reg, n)
    if case["measure"]:
        out.update(_measured(s, reg))
    return out


# ---- the work of a pass -----------------------------------------------------

def work(case):
    """Bytes: every register in hand read once, every fresh register written
    once and read once for its results.  Flops: one complex multiply-add (8)
    per amplitude a one-qubit gate changes, FP products of the density."""
    kind = case["kind"]
    amp = 16 if case["precision"] == 2 else 8
    if kind == "batch":
        ns = range(case["qmin"], case["qmax"] + 1)
        each = case["count"] / len(ns)
        depth = (case["dmin"] + case["dmax"]) / 2
        flops = sum(each * depth * 8 * (n + (n // 2) / 2) * 2.0 ** n + each * 4 * 2.0 ** (n + n // 2)
                    for n in ns)
        return {"bytes": sum(each * 16 * 4.0 ** (n // 2) for n in ns), "flops": flops}
    if kind == "join":
        size = 2.0 ** (case["most"] + case["least"])
        return {"bytes": amp * (2.0 ** case["most"] + 2.0 ** case["least"] + 2 * size),
                "flops": 6 * size}
    n = case["n"]
    size = 2.0 ** n
    if kind == "measure":
        return {"bytes": amp * size * (1 + 2.0 ** -case["measure"]), "flops": 3 * size}
    if kind == "density":
        return {"bytes": amp * size + 16 * 4.0 ** case["keep"],
                "flops": 4 * size * 2.0 ** case["keep"]}
    if kind == "steps":
        return {"bytes": amp * size * (2 * case["gates"]), "flops": 8 * size * case["gates"]}
    if case["family"] == "layers":
        per_layer = n + 0.5 * (n // 2) + 0.25
    else:
        per_layer = n + 0.5 * ((n - 1) / 2)
    flops = 8 * size * per_layer * case["depth"]
    nbytes = 2 * amp * size
    if case["amps"]:
        nbytes += 16 * size
    if case["keep"]:
        flops += 4 * size * 2.0 ** case["keep"]
        nbytes += 16 * 4.0 ** case["keep"]
    return {"bytes": nbytes, "flops": flops}


# ---- 64-bit values, in plain torch -----------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _split(psi, n, qubits):
    """psi as a view with a dimension of 2 for each of `qubits` (highest first)."""
    qs = sorted(qubits, reverse=True)
    shape, prev = [], n
    for q in qs:
        shape += [1 << (prev - q - 1), 2]
        prev = q
    shape.append(1 << prev)
    return psi.view(shape), {q: 2 * i + 1 for i, q in enumerate(qs)}


def _pick(view, dims, values):
    idx = [slice(None)] * view.dim()
    for q, v in values.items():
        idx[dims[q]] = v
    return view[tuple(idx)]


def _one(psi, n, op):
    """A controlled one-qubit gate, in place."""
    t = op.targets[0]
    view, dims = _split(psi, n, {t} | op.controls | op.anticontrols)
    on = {q: 1 for q in op.controls}
    on.update({q: 0 for q in op.anticontrols})
    x0, x1 = _pick(view, dims, {**on, t: 0}), _pick(view, dims, {**on, t: 1})
    m = [[complex(v) for v in row] for row in np.asarray(op.gate)]
    if m == [[1, 0], [0, -1]]:
        x1.neg_()
        return
    y0 = x0 * m[0][0] + x1 * m[0][1]
    y1 = x0 * m[1][0] + x1 * m[1][1]
    x0.copy_(y0)
    x1.copy_(y1)


def _products(psi, n, mats):
    """2x2 matrices on separate qubits, five neighbouring qubits to a product."""
    for lo in range(0, n, 5):
        qs = [q for q in range(lo, min(lo + 5, n))]
        if not any(q in mats for q in qs):
            continue
        k = np.eye(1, dtype=np.complex128)
        for q in qs:
            k = np.kron(mats.get(q, np.eye(2)), k)
        k = torch.from_numpy(k).to(psi.device)
        dim = 1 << len(qs)
        if lo == 0:
            psi = (psi.view(-1, dim) @ k.T).reshape(-1)
        else:
            psi = torch.matmul(k, psi.view(-1, dim, 1 << lo)).reshape(-1)
    return psi


def _evolve(psi, n, ops):
    mats = {}
    for op in ops:
        if not op.controls and not op.anticontrols:
            q = op.targets[0]
            mats[q] = np.asarray(op.gate) @ mats.get(q, np.eye(2))
            continue
        if any(q in mats for q in set(op.targets) | op.controls | op.anticontrols):
            psi = _products(psi, n, mats)
            mats = {}
        _one(psi, n, op)
    return _products(psi, n, mats)


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=_device())
    psi[0] = 1
    return psi


def _norm2(x):
    return float(torch.view_as_real(x.contiguous()).square().sum())


def _exact_probs(psi, n):
    w = torch.view_as_real(psi.contiguous()).square().sum(-1)
    return [float(w.view(-1, 2, 1 << q)[:, 1].sum() / w.sum()) for q in range(n)]


def _exact_measured(psi, n, mask, rolls):
    out, i, cur = [], 0, n
    for q in range(n - 1, -1, -1):
        if not (mask >> q) & 1:
            out.append(-1)
            continue
        view, dims = _split(psi, cur, {q})
        p = _norm2(_pick(view, dims, {q: 1})) / _norm2(psi)
        bit = 1 if p > rolls[i] else 0
        i += 1
        out.append(bit)
        psi = _pick(view, dims, {q: bit}).contiguous().reshape(-1)
        cur -= 1
    got = {"outcomes": np.array(out, dtype=np.int64)}
    if cur:
        got["left"] = np.array(_exact_probs(psi, cur))
    return got


def _exact_density(psi, n, keep):
    view, dims = _split(psi, n, range(n))
    if keep == list(range(len(keep))):
        x = psi.view(-1, 1 << len(keep))
    else:
        traced = [q for q in range(n - 1, -1, -1) if q not in keep]
        order = [dims[q] for q in traced] + [dims[q] for q in reversed(keep)]
        rest = [i for i in range(view.dim()) if i not in order]
        x = view.permute(order + rest).reshape(-1, 1 << len(keep))
    rho = x.T @ x.conj()
    return (rho / _norm2(psi)).cpu().numpy()


def _exact_batch(case, seed):
    """All circuits of one width together: gate i of each, element by element."""
    flat = _batch(case, seed)
    dev = _device()
    rhos = [None] * flat.count
    for n in sorted(set(int(x) for x in flat.num_qubits)):
        cs = [c for c in range(flat.count) if int(flat.num_qubits[c]) == n]
        steps = max(int(flat.op_start[c + 1] - flat.op_start[c]) for c in cs)
        tg = np.zeros((steps, len(cs)), dtype=np.int64)
        cm = np.zeros((steps, len(cs)), dtype=np.int64)
        mat = np.zeros((steps, len(cs), 4), dtype=np.complex128)
        mat[:, :, 0] = mat[:, :, 3] = 1
        for j, c in enumerate(cs):
            a, b = int(flat.op_start[c]), int(flat.op_start[c + 1])
            tg[:b - a, j] = flat.op_targets[a:b, 0]
            cm[:b - a, j] = flat.op_controls[a:b].astype(np.int64)
            mat[:b - a, j] = flat.matrices[flat.op_matrix[a:b].astype(np.int64)[:, None] +
                                           np.arange(4)]
        tg, cm, mat = (torch.from_numpy(x).to(dev) for x in (tg, cm, mat))
        i = torch.arange(1 << n, device=dev)[None, :]
        psi = torch.zeros(len(cs), 1 << n, dtype=torch.complex128, device=dev)
        psi[:, 0] = 1
        for g in range(steps):
            t, c, m = tg[g][:, None], cm[g][:, None], mat[g]
            bit = (i >> t) & 1
            other = torch.gather(psi, 1, i ^ (1 << t))
            own = torch.where(bit == 1, m[:, 3:4], m[:, 0:1])
            off = torch.where(bit == 1, m[:, 2:3], m[:, 1:2])
            psi = torch.where((i & c) == c, own * psi + off * other, psi)
        for j, c in enumerate(cs):
            x = psi[j].view(-1, 1 << int(flat.keep[c]))
            rhos[c] = ((x.T @ x.conj()) / _norm2(psi[j])).reshape(-1)
    return torch.cat(rhos).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "join":
        rng = _rng(case, seed)
        a = _evolve(_zero(case["most"]), case["most"], _random_layer(rng, case["most"]))
        b = _evolve(_zero(case["least"]), case["least"], _random_layer(rng, case["least"]))
        return np.array(_exact_probs(torch.outer(a, b).reshape(-1),
                                     case["most"] + case["least"]))
    n = case["n"]
    mask, rolls, keep = _ending(case, seed, n)
    if kind == "circuit":
        psi = _evolve(_zero(n), n, _ops(case, seed))
        out = {"probs": np.array(_exact_probs(psi, n))}
        if case["amps"]:
            out["amps"] = (psi / math.sqrt(_norm2(psi))).cpu().numpy()
        if case["keep"]:
            out["rho"] = _exact_density(psi, n, keep)
        if case["measure"]:
            out.update(_exact_measured(psi, n, mask, rolls))
        return out
    psi = _evolve(_zero(n), n, _random_layer(_rng(case, seed), n))
    if kind == "measure":
        return _exact_measured(psi, n, mask, rolls)
    if kind == "density":
        return _exact_density(psi, n, keep)
    probs = []
    for op in _step_ops(case, seed):
        psi = _evolve(psi, n, [op])
        view, dims = _split(psi, n, {op.targets[0]})
        probs.append(_norm2(_pick(view, dims, {op.targets[0]: 1})) / _norm2(psi))
    return {"after_each": np.array(probs), "probs": np.array(_exact_probs(psi, n))}

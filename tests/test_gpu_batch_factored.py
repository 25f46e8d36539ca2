"""Batches of factored circuits on the GPU against the oracle: one-tile registers
below and above a warp, clusters of 2 to 8 CTAs (also with tiles too narrow to fill a
warp), matrices over no qubit, one and many, circuits without gates, and dense
2-qubit circuits, which run gate by gate, between them."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.conftest import ATOL_C128, ATOL_C64
from tests.test_plan import random_ops
from tests.test_plan_factored import one_qubit_ops

pytestmark = pytest.mark.gpu


def flat_batch(circuits):
    """[(qubits, keep, ops)] as a FlatBatch."""
    ops = [op for _, _, o in circuits for op in o]
    tg = np.zeros((len(ops), 3), dtype=np.uint32)
    for i, op in enumerate(ops):
        tg[i, :op.k] = op.targets
    mats = [np.asarray(op.gate, dtype=np.complex128).reshape(-1) for op in ops]
    sizes = [m.size for m in mats]
    return W.FlatBatch(
        num_qubits=np.array([c[0] for c in circuits], dtype=np.uint32),
        keep=np.array([c[1] for c in circuits], dtype=np.uint32),
        op_start=np.cumsum([0] + [len(c[2]) for c in circuits]).astype(np.uint64),
        op_k=np.array([op.k for op in ops], dtype=np.uint32),
        op_targets=tg,
        op_controls=np.array([sum(1 << q for q in op.controls) for op in ops], dtype=np.uint64),
        op_anticontrols=np.array([sum(1 << q for q in op.anticontrols) for op in ops],
                                 dtype=np.uint64),
        op_matrix=np.cumsum([0] + sizes[:-1]).astype(np.uint64),
        matrices=np.concatenate(mats))


@pytest.mark.parametrize("keep_states", [True, False])
@pytest.mark.parametrize("precision,tile_bits", [(2, 12), (1, 12), (2, 8), (1, 9)])
def test_factored_circuits(dk_gpu, orc, precision, tile_bits, keep_states):
    from doki_b200.batch import BatchEngine

    circuits = []
    for i, n in enumerate([4, 5, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16]):
        for j, keep in enumerate(sorted({0, 1, n // 2, min(n, 9)})):
            ops = one_qubit_ops(W.rng_for(900 + 10 * i + j), n, 20 + 10 * j)
            circuits.append((n, keep, ops))
        circuits.append((n, 2, []))
        circuits.append((n, 2, [W.Op(W.H.copy(), [q]) for q in range(n)]
                         + random_ops(W.rng_for(990 + i), n, 12, kmax=2)))
    eng = BatchEngine(flat_batch(circuits), precision=precision, tile_bits=tile_bits)
    eng.run(keep_states=keep_states)
    eng.sync()
    atol = ATOL_C128 if precision == 2 else ATOL_C64
    for c, (n, keep, ops) in enumerate(circuits):
        psi = orc.registry_get_all(W.run_ops(orc, orc.registry_new(n), ops))
        if keep_states:
            got = eng.state(c)
            assert np.allclose(got / np.linalg.norm(got), psi, atol=atol, rtol=0), (c, n)
        x = np.asarray(psi).reshape(1 << (n - keep), 1 << keep)
        assert np.allclose(eng.rho(c), x.T @ x.conj(), atol=atol, rtol=0), (c, n, keep)
    eng.close()

"""Layers of Ry and CNOTs on the GPU against the oracle: real rotations share stages
with the CNOTs as relabellings, in sweeps and in batches."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.conftest import ATOL_C128, ATOL_C64
from tests.test_gpu_batch_factored import flat_batch
from tests.test_plan_real_gates import ry

pytestmark = pytest.mark.gpu


def ansatz(n, layers, seed):
    rng = W.rng_for(seed)
    ops = []
    for layer in range(layers):
        ops += [W.Op(ry(rng.uniform(0, 6)), [q]) for q in range(n)]
        pairs = [(q, (q + 1) % n) for q in range(n)]
        for c, t in pairs if layer % 2 else [p[::-1] for p in reversed(pairs)]:
            ops.append(W.Op(W.X.copy(), [t], {c}))
    return ops


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n", [4, 6, 9, 12, 14, 17])
def test_sweeps(dk_gpu, orc, n, prec):
    tol = ATOL_C128 if prec == 2 else ATOL_C64
    for seed in range(6):
        ops = ansatz(n, 5, 9000 + 10 * n + seed)
        got = dk_gpu.registry_get_all(W.run_ops(dk_gpu, dk_gpu.registry_new(n, False, prec), ops), False)
        want = orc.registry_get_all(W.run_ops(orc, orc.registry_new(n), ops))
        assert np.allclose(got, want, atol=tol, rtol=0), seed


@pytest.mark.parametrize("prec", [2, 1])
def test_batches(dk_gpu, orc, prec):
    from doki_b200.batch import BatchEngine

    circuits = [(n, 2, ansatz(n, 4, 9100 + 10 * n + i)) for n in range(4, 17) for i in range(3)]
    eng = BatchEngine(flat_batch(circuits), precision=prec)
    eng.run(keep_states=True)
    eng.sync()
    tol = ATOL_C128 if prec == 2 else ATOL_C64
    for c, (n, _, ops) in enumerate(circuits):
        want = orc.registry_get_all(W.run_ops(orc, orc.registry_new(n), ops))
        got = eng.state(c)
        assert np.allclose(got / np.linalg.norm(got), want, atol=tol, rtol=0), (c, n)
    eng.close()

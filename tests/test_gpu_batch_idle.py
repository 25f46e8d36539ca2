"""Batches whose circuits have passes with nothing to do (controlled phases of angle
0, CNOTs that undo each other), on the GPU against the oracle: 10 to 12 qubits, where
several warps share a register."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.conftest import ATOL_C128, ATOL_C64
from tests.test_gpu_batch_factored import flat_batch
from tests.test_plan_barriers import equal_pairs, phases_of_angle_0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [2, 1])
def test_idle_passes(dk_gpu, orc, precision):
    from doki_b200.batch import BatchEngine

    circuits = [(n, 3, make(n, seed)) for n in (10, 11, 12) for seed in range(6)
                for make in (phases_of_angle_0, equal_pairs)]
    eng = BatchEngine(flat_batch(circuits * 8), precision=precision)
    eng.run(keep_states=True)
    eng.sync()
    atol = ATOL_C128 if precision == 2 else ATOL_C64
    for c, (n, _, ops) in enumerate(circuits):
        psi = orc.registry_get_all(W.run_ops(orc, orc.registry_new(n), ops))
        for copy in range(8):
            got = eng.state(c + copy * len(circuits))
            assert np.allclose(got / np.linalg.norm(got), psi, atol=atol, rtol=0), (c, n, copy)
    eng.close()

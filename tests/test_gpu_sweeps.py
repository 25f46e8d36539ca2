"""Factored sweeps on the GPU against the oracle: every tile width, controls in
and off a pass and outside the tile, tiles that no gate acts on, programs cut at
their size limit, and gates that need the other sweeps among them."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.conftest import ATOL_C128, ATOL_C64
from tests.test_plan import random_ops
from tests.test_plan_factored import one_qubit_ops

pytestmark = pytest.mark.gpu


def check(d, orc, n, prec, ops, seed):
    rng = W.rng_for(seed)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    a = W.run_ops(d, d.registry_new_data(n, psi, 0, prec), ops)
    b = W.run_ops(orc, orc.registry_new_data(n, psi), ops)
    tol = ATOL_C128 if prec == 2 else ATOL_C64
    assert np.allclose(d.registry_get_all(a, False), orc.registry_get_all(b), atol=tol, rtol=0)
    assert np.allclose(d.registry_probs(a), orc.registry_probs(b), atol=tol, rtol=0)


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n", [4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 17])
def test_gates_with_controls_everywhere(dk_gpu, orc, n, prec):
    check(dk_gpu, orc, n, prec, one_qubit_ops(W.rng_for(300 + n), n, 100), 310 + n)


@pytest.mark.parametrize("prec", [2, 1])
def test_tiles_that_no_gate_acts_on(dk_gpu, orc, prec):
    """Sweeps in which every gate depends on qubits outside the tile run in
    place and skip the other tiles; the norm stays exact (non-unitary gates
    change it)."""
    n = 17
    rng = W.rng_for(320)
    reg, ref = dk_gpu.registry_new(n, False, prec), orc.registry_new(n)
    ops = [W.Op(W.H.copy(), [q]) for q in range(n)]
    for rep in range(4):
        for q in range(3):
            ops.append(W.Op(W.u3(*rng.uniform(0, 6, 3)), [q], {16}, {15}))
            ops.append(W.Op(np.array([[1.0, 0.25], [-0.5, 1.25]], dtype=complex), [q + 4], {14 + rep % 2}))
        reg = W.run_ops(dk_gpu, reg, ops)
        ref = W.run_ops(orc, ref, ops)
        tol = ATOL_C128 if prec == 2 else ATOL_C64
        assert np.allclose(dk_gpu.registry_probs(reg), orc.registry_probs(ref), atol=tol, rtol=0)
        assert np.allclose(dk_gpu.registry_get_all(reg, False), orc.registry_get_all(ref),
                           atol=tol, rtol=0)
        ops = []


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n", [12, 20])
def test_long_programs(dk_gpu, orc, n, prec):
    """Several hundred gates on few qubits: the program is cut at its limit
    (a longer one for a register of few tiles)."""
    rng = W.rng_for(330 + n)
    ops = []
    for _ in range(400):
        q = int(rng.integers(0, 6))
        far = {int(n - 1 - rng.integers(0, 3))} if rng.random() < 0.4 else set()
        ops.append(W.Op(W.u3(*rng.uniform(0, 6, 3)), [q], far))
    check(dk_gpu, orc, n, prec, ops, 340 + n)


@pytest.mark.parametrize("prec", [2, 1])
def test_other_sweeps_in_between(dk_gpu, orc, prec):
    n = 14
    rng = W.rng_for(350)
    ops = []
    for _ in range(6):
        ops += one_qubit_ops(rng, n, 20) + random_ops(rng, n, 10)
    check(dk_gpu, orc, n, prec, ops, 351)


@pytest.mark.parametrize("prec", [2, 1])
def test_norm_between_measurements(dk_gpu, orc, prec):
    """The blocks of a sweep count themselves down to the last, which makes the
    norm, in a scratch that measurements use too: flushes of 1 to 32 blocks with
    joint measurements in between."""
    for n in (12, 13, 17, 14):
        rng = W.rng_for(340 + n)
        mask = sum(1 << int(q) for q in rng.permutation(n)[:3])
        reg = W.run_ops(dk_gpu, dk_gpu.registry_new(n, False, prec), one_qubit_ops(rng, n, 20))
        for _ in range(3):
            left, _ = dk_gpu.registry_measure(reg, mask, [0.3, 0.6, 0.9], -1, False)
            assert abs(np.linalg.norm(dk_gpu.registry_get_all(left, False)) - 1) < 1e-5
            reg = W.run_ops(dk_gpu, reg, one_qubit_ops(rng, n, 10))
            assert abs(np.linalg.norm(dk_gpu.registry_get_all(reg, False)) - 1) < 1e-5

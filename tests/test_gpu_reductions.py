"""Marginals and the joint distribution of measured qubits at the edges of their
kernels' blocks, against plain numpy sums of the register's own amplitudes."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W

pytestmark = pytest.mark.gpu


def register(d, n, prec, seed):
    rng = W.rng_for(seed)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    reg = d.registry_new_data(n, psi / np.linalg.norm(psi), 0, prec)
    return reg, np.asarray(d.registry_get_all(reg, False)), rng


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n", [1, 4, 5, 7, 8, 9, 12, 13, 17, 20])
def test_marginals_of_every_block_shape(dk_gpu, n, prec):
    """One warp with idle lanes up to the full grid.  Both sides add the same
    2^n FP64 squares in another order: within 2^n * eps at worst, far less
    pairwise; 1e-13 is above sqrt(2^20) * eps."""
    reg, amps, _ = register(dk_gpu, n, prec, 40 + n)
    w = np.abs(amps) ** 2
    want = [w.reshape(-1, 2, 1 << q)[:, 1].sum() for q in range(n)]
    assert np.allclose(dk_gpu.registry_probs(reg), want, atol=1e-13, rtol=0)


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n,mask", [
    (3, 0b101), (8, 0b10000001), (9, 0b100000000), (12, 0xfff), (12, 0b100000000001),
    (13, 0b1100000000000), (15, 0x0fff), (15, 0x7ff8), (16, 0b1001100000010001),
    (18, 0b110000), (18, 0x3f00), (20, 0xff000)])
def test_joint_measurement_at_chunk_edges(dk_gpu, n, mask, prec):
    """Measured qubits inside, across and above the 12-bit chunks a block
    reads: outcomes follow the sequential rule on numpy sums (rolls away from
    every decision by 1e-9), and the collapsed register is the selected
    amplitudes over their norm."""
    reg, amps, rng = register(dk_gpu, n, prec, 70 + n)
    qs = [q for q in range(n - 1, -1, -1) if (mask >> q) & 1]
    idx = np.arange(1 << n)
    left, p = np.ones(1 << n, dtype=bool), np.abs(amps) ** 2
    rolls, want = [], []
    for q in qs:
        p1 = p[left & ((idx >> q) & 1 == 1)].sum() / p[left].sum()
        roll = rng.random()
        while abs(roll - p1) < 1e-9:
            roll = rng.random()
        bit = 1 if p1 > roll else 0
        rolls.append(roll)
        want.append(bit)
        left &= (idx >> q) & 1 == bit
    after, res = dk_gpu.registry_measure(reg, mask, rolls, 1, False)
    assert [int(v) for v in res if v is not None] == want
    if after is None:
        assert len(qs) == n
        return
    sel = amps[left]
    assert np.allclose(dk_gpu.registry_get_all(after, False), sel / np.linalg.norm(sel),
                       atol=1e-12, rtol=0)

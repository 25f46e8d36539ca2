"""Reduced density matrices on the GPU against a plain product of the gathered
amplitudes: kept qubits low, high and scattered (the gather's tiles then take
from 5 to 10 index bits), registers smaller than a tile, traced ranges that do and
do not fill their splits."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.conftest import ATOL_C128, ATOL_C64

pytestmark = pytest.mark.gpu


def product(psi, n, kept):
    rest = [q for q in range(n) if q not in kept]
    idx = np.arange(1 << n)
    a = sum(((idx >> q) & 1) << j for j, q in enumerate(kept))
    b = sum(((idx >> q) & 1) << j for j, q in enumerate(rest)) if rest else 0 * idx
    x = np.empty((1 << len(rest), 1 << len(kept)), dtype=np.complex128)
    x[b, a] = psi
    return x.T @ x.conj()


@pytest.mark.parametrize("prec", [2, 1])
@pytest.mark.parametrize("n,k", [(1, 1), (3, 2), (5, 3), (9, 5), (10, 6), (11, 3), (13, 7), (14, 8),
                                 (15, 6), (16, 7), (17, 8), (17, 9)])
def test_kept_anywhere(dk_gpu, n, k, prec):
    rng = W.rng_for(700 + 10 * n + k)
    psi = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    psi /= np.linalg.norm(psi)
    reg = dk_gpu.registry_new_data(n, psi, 0, prec)
    sets = [list(range(k)), list(range(n - k, n)), list(range(0, n, 2))[:k] + list(range(1, n, 2))]
    sets += [rng.permutation(n).tolist() for _ in range(3)]
    tol = ATOL_C128 if prec == 2 else ATOL_C64
    for s in sets:
        kept = sorted(s[:k])
        rho = dk_gpu.registry_density(reg, False)
        for q in range(n - 1, -1, -1):
            if q not in kept:
                rho = dk_gpu.funmatrix_partialtrace(rho, q, False)
        assert np.allclose(dk_gpu.funmatrix_numpy(rho), product(psi, n, kept), atol=tol, rtol=0), kept


@pytest.mark.parametrize("n,k", [(22, 7), (21, 8), (22, 8), (20, 9), (20, 10), (21, 11)])
def test_large_complex64(dk_gpu, n, k):
    """Products of 8-bit digits (complex64, at least 128 kept indices, 1024
    traced ones and 2^29 products): rows of very different size, an empty one, and amplitudes far
    below their row's largest.  Every entry within 2^-16 of its rows' norms: the
    digits' error is at most 2^-33 of the rows' largest products per traced index
    (here up to 2^15), the register's rounding 2^-24 of each amplitude."""
    rng = W.rng_for(800 + 10 * n + k)
    for kept in (list(range(k)), sorted(rng.permutation(n)[:k].tolist())):
        rest = [q for q in range(n) if q not in kept]
        idx = np.arange(1 << n)
        a = sum(((idx >> q) & 1) << j for j, q in enumerate(kept))
        b = sum(((idx >> q) & 1) << j for j, q in enumerate(rest))
        psi = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)) * 2.0 ** -(a % 13)
        psi *= np.where(b % 5 == 0, 2.0 ** -9, 1.0) * (a != 3)
        psi = (psi / np.linalg.norm(psi)).astype(np.complex64).astype(np.complex128)
        reg = dk_gpu.registry_new_data(n, psi, 0, 1)
        rho = dk_gpu.registry_density(reg, False)
        for q in range(n - 1, -1, -1):
            if q not in kept:
                rho = dk_gpu.funmatrix_partialtrace(rho, q, False)
        got, want = dk_gpu.funmatrix_numpy(rho), product(psi, n, kept)
        size = np.sqrt(np.diag(want).real)
        assert (np.abs(got - want) <= 2.0 ** -16 * np.outer(size, size)).all(), kept
        assert np.array_equal(got, got.conj().T)

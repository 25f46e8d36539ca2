"""Small entries of reduced density matrices on the GPU.  Each row of the register
(kept index) has one dominant amplitude, at a traced index where every other row is
0, so that an entry off the diagonal is a sum of products of the others only: 1e-8
or 1e-12 of the rows' largest.  FP64 sums keep their digits."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.test_gpu_density import product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("n,k,small", [(22, 7, 1e-4), (22, 7, 1e-6), (21, 8, 1e-6), (20, 9, 1e-4),
                                       (14, 6, 1e-6)])
def test_entries_beside_dominant_amplitudes(dk_gpu, n, k, small, prec):
    """Worst case of a sum of K = 2^(n - k) FP64 products in any order: K 2^-53 of
    the sum of their magnitudes, for each of the two sides."""
    rng = W.rng_for(850 + 10 * n + k)
    dim, K = 1 << k, 1 << (n - k)
    for kept in (list(range(k)), sorted(rng.permutation(n)[:k].tolist())):
        rest = [q for q in range(n) if q not in kept]
        x = (rng.normal(size=(K, dim)) + 1j * rng.normal(size=(K, dim))) * small
        # row a is dominant at traced index a mod K; below 2^k such indices are shared
        at = rng.permutation(K)[:dim] if K >= dim else np.arange(dim) % K
        x[at, :] = 0
        x[at, np.arange(dim)] = np.exp(2j * np.pi * rng.random(dim))
        x = x.astype(np.complex64).astype(np.complex128)
        idx = np.arange(1 << n)
        a = sum(((idx >> q) & 1) << j for j, q in enumerate(kept))
        b = sum(((idx >> q) & 1) << j for j, q in enumerate(rest))
        psi = x[b, a]
        reg = dk_gpu.registry_new_data(n, psi, 0, prec)
        rho = dk_gpu.registry_density(reg, False)
        for q in range(n - 1, -1, -1):
            if q not in kept:
                rho = dk_gpu.funmatrix_partialtrace(rho, q, False)
        got = dk_gpu.funmatrix_numpy(rho)
        # data registers are taken as they are, normalised or not
        want, size = product(psi, n, kept), np.abs(x).T @ np.abs(x)
        assert (np.abs(got - want) <= (2 * K + 64) * 2.0 ** -53 * size).all(), kept

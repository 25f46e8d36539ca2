"""Many large gate matrices in one flush: they pass through a ring of two 1 MiB
parts on their way to the device while the gates before them run.  8-qubit matrices
fill a part exactly, 7- and 4-qubit ones after 4 and 256, 9-qubit ones are longer
than a part.  Compared with the same
gates flushed one at a time (the same kernels on the same data: equal to the last
bit)."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.golden.gen_golden import random_unitary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,count", [(24, 8, 7), (22, 7, 20), (20, 4, 600), (20, 9, 6)])
def test_matrices_in_one_flush(dk_gpu, n, k, count):
    d = dk_gpu
    rng = W.rng_for(60 + k)
    some = [random_unitary(rng, k) for _ in range(min(count, 12))]
    # the same matrix never follows itself two parts later
    ops = []
    for i in range(count):
        m = some[i % len(some)] * np.exp(1j * rng.random())
        ops.append(W.Op(m, [int(q) for q in rng.permutation(n)[:k]]))
    start = W.run_ops(d, d.registry_new(n, False), [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q])
                                                    for q in range(n)])
    d.registry_flush(start)
    one = W.run_ops(d, start, ops)
    each = start
    for op in ops:
        each = W.run_ops(d, each, [op])
        d.registry_flush(each)
    a, b = (np.asarray(d.registry_get_all(r, False)) for r in (one, each))
    assert np.array_equal(a, b)

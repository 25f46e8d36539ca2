"""A flush whose memory cannot be had leaves the register as it was: sweeps run in
place, so everything that any step needs is allocated before the first one.  A child
process with a device-memory budget that a second register of the same size fills."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import numpy as np
import doki_b200
from doki_b200 import workloads as W
from tests.golden.gen_golden import random_unitary

d = doki_b200.load()
n, k = 20, %d
rng = W.rng_for(5)
first = [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q]) for q in range(n)]
then = [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q]) for q in range(n)]
then += [W.Op(random_unitary(rng, k), [int(q) for q in rng.permutation(n)[:k]])]
then += [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q]) for q in range(n)]

def fresh():
    reg = W.run_ops(d, d.registry_new(n, False), first)
    d.registry_flush(reg)
    return reg

want = np.asarray(d.registry_probs(W.run_ops(d, fresh(), then)))
reg = fresh()
reg = W.run_ops(d, reg, then)  # the only owner of its buffer: it runs in place
other = fresh()
for _ in range(3):
    try:
        d.registry_probs(reg)
        raise SystemExit("the flush found memory")
    except SystemExit:
        raise
    except Exception as e:
        assert "budget" in str(e) or "alloc" in str(e).lower(), e
d.registry_del(other, False)
got = np.asarray(d.registry_probs(reg))
assert np.array_equal(got, want), np.abs(got - want).max()
print("intact")
"""


@pytest.mark.parametrize("k", [4, 9])
def test_register_survives(k):
    """No room for the output of a gate that no sweep runs (9 qubits: with a matrix
    that is too long for staging)."""
    size = 16 << 20
    env = dict(os.environ, DK_HBM_BUDGET_BYTES=str(11 * size // 4), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD % k], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "intact", r.stdout + r.stderr[-2000:]

"""Circuits of dense 2-qubit gates on large complex64 registers: as many sweeps as
their planner makes of them by itself."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.conftest import ATOL_C64
from tests.test_plan_low_bits import brickwork

pytestmark = pytest.mark.gpu


def test_dense_brickwork(dk_gpu):
    d, n = dk_gpu, 24
    ops = brickwork(n, 20, n)
    before = d.engine_stats()["sweeps"]
    reg = W.run_ops(d, d.registry_new(n, False, 1), ops)
    d.registry_flush(reg)
    assert d.engine_stats()["sweeps"] - before == 21
    want = W.run_ops(d, d.registry_new(n, False, 2), ops)
    assert np.allclose(d.registry_probs(reg), d.registry_probs(want), atol=ATOL_C64, rtol=0)

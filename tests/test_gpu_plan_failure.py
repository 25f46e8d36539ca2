"""A plan that fails on the way, on the GPU: the gates that have run stay done and the
others are queued again, so that the register is the one that was asked for and the
next read goes on.  Child processes in which the planner of dense gates is made to
fail at its n-th call (a shim in front of the library)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <string.h>
#include "dk_internal.h"
static int until = -1;
void fail_plan_at(int call) { until = call; }
int dk_plan_build(const dk_flat_op *ops, int nops, unsigned n, int prec,
		  const dk_plan_limits *lim, dk_plan *plan)
{
	static int (*real)(const dk_flat_op *, int, unsigned, int, const dk_plan_limits *, dk_plan *);
	if (!real)
		real = dlsym(RTLD_NEXT, "dk_plan_build");
	if (until >= 0 && until-- == 0) {
		memset(plan, 0, sizeof(*plan));
		return DK_ERR_ALLOC;
	}
	return real(ops, nops, n, prec, lim, plan);
}
"""

CHILD = r"""
import ctypes, os
import numpy as np
import doki_b200
from doki_b200 import workloads as W
from tests.golden.gen_golden import random_unitary

d = doki_b200.load()
shim = ctypes.CDLL(os.environ["LD_PRELOAD"].split()[0])
for n, prec in ((16, 2), (16, 1), (12, 2)):
    rng = W.rng_for(n + prec)
    ops = []
    for layer in range(6):
        ops += [W.Op(W.u3(*rng.uniform(0, 6, 3)), [q]) for q in range(n)]
        for _ in range(4):
            q = [int(x) for x in rng.permutation(n)]
            ops.append(W.Op(random_unitary(rng, 2), q[:2], {q[2]} if rng.random() < 0.5 else set()))
        ops.append(W.Op(W.X.copy(), [layer], {layer + 1}))
    ops.insert(40, W.Op(random_unitary(rng, 4), [0, 5, 3, 8]))
    want = np.asarray(d.registry_get_all(W.run_ops(d, d.registry_new(n, False, prec), ops), False))
    tol = 1e-12 if prec == 2 else 5e-5
    failed = 0
    for shared in (False, True):
        for call in range(12):
            reg = W.run_ops(d, d.registry_new(n, False, prec), ops[:n])
            d.registry_flush(reg)
            first = reg if shared else None  # another register on the same buffer
            before = np.asarray(d.registry_get_all(reg, False)) if shared else None
            reg = W.run_ops(d, reg, ops[n:])
            shim.fail_plan_at(call)
            try:
                d.registry_flush(reg)
            except Exception as e:
                failed += 1
                assert "alloc" in str(e).lower(), e
                if call % 2:  # a second failure on the way
                    shim.fail_plan_at(1)
                    try:
                        d.registry_flush(reg)
                    except Exception:
                        failed += 1
            shim.fail_plan_at(-1)
            more = W.run_ops(d, reg, [W.Op(W.H.copy(), [0])] * 2)  # gates behind those left
            for r in (reg, more):
                got = np.asarray(d.registry_get_all(r, False))
                assert np.allclose(got, want, atol=tol, rtol=0), (n, prec, call)
            if shared:
                assert np.array_equal(np.asarray(d.registry_get_all(first, False)), before)
    assert failed > 5, failed  # the shim reached the plans
print("ok")
"""


def test_gates_that_are_left_run_later(tmp_path):
    src, lib = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    r = subprocess.run([shutil.which("gcc") or "/usr/bin/gcc", "-std=gnu11", "-shared", "-fPIC",
                        "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "doki_b200", "csrc"),
                        "-I", "/usr/local/cuda/include", str(src), "-ldl", "-o", str(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    # the library behind the shim, for its RTLD_NEXT
    engine = os.path.join(ROOT, "doki_b200", "libdokigpu.so")
    env = dict(os.environ, LD_PRELOAD=f"{lib} {engine}", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr[-2000:]

"""Planning of a batch circuit (doki_b200/csrc/dk_batch_plan.h), on CPU against a
planner that answers as it is told: the kernels of factored circuits take every
program they are given for a factored one, so a step of any other kind has to send
the circuit to the gate-by-gate kernel, with nothing left of its plan."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

DRIVER = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "dk_batch_plan.h"

/* steps by letter: f factored, t tensor, s scalar, g generic gate, e failure */
static const char *script;
static int all = 1, ended = 0;
static unsigned char program[256];

extern "C" {
void dk_plan_default_limits(int, unsigned, dk_plan_limits *) {}
int dk_fx_begin(const dk_flat_op *, int, unsigned, int, const dk_plan_limits *, dk_fx_plan **out)
{
	*out = (dk_fx_plan *)program;
	return DK_OK;
}
int dk_fx_all(const dk_fx_plan *) { return all; }
void dk_fx_end(dk_fx_plan *) { ended++; }
int dk_fx_next(dk_fx_plan *, dk_step *step, const unsigned char **prog)
{
	const char c = *script;
	if (!c)
		return 0;
	script++;
	if (c == 'e')
		return -DK_ERR_ALLOC;
	memset(step, 0, sizeof(*step));
	step->kind = c == 'g' ? 2 : 1;
	dk_sweep_hdr *h = (dk_sweep_hdr *)program;
	memset(program, 0, sizeof(program));
	h->mode = c == 'f' ? DK_SWEEP_FACTORED : c == 't' ? DK_SWEEP_TENSOR : DK_SWEEP_SCALAR;
	h->bytes = sizeof(dk_sweep_hdr);
	*prog = c == 'g' ? nullptr : program;
	return 1;
}
}

int main(int argc, char **argv)
{
	script = argv[1];
	all = atoi(argv[2]);
	dk::BatchProgram p;
	int rc = -1;
	std::vector<dk_flat_op> none;
	const int other = dk::plan_factored(none, 12, DK_C128, 12, &p, &rc);
	printf("%d %d %u %zu %d\n", other, rc, p.nsweep, p.bytes.size() / sizeof(dk_sweep_hdr), ended);
	return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("batch_plan")
    src, exe = tmp / "driver.cpp", tmp / "driver"
    src.write_text(DRIVER)
    r = subprocess.run([shutil.which("g++") or "/usr/bin/g++", "-std=c++17", "-O1",
                        "-I", os.path.join(ROOT, "include"),
                        "-I", os.path.join(ROOT, "doki_b200", "csrc"),
                        "-I", "/usr/local/cuda/include", str(src), "-o", str(exe), "-ldl"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(exe)


@pytest.mark.parametrize("script,all_factor,want", [
    ("", 1, [0, 0, 0, 0, 1]),
    ("fff", 1, [0, 0, 3, 3, 1]),
    ("fff", 0, [1, 0, 0, 0, 1]),
    ("t", 1, [1, 0, 0, 0, 1]),
    ("ffs", 1, [1, 0, 0, 0, 1]),
    ("fg", 1, [1, 0, 0, 0, 1]),
])
def test_other_steps_leave_nothing(driver, script, all_factor, want):
    out = subprocess.run([driver, script, str(all_factor)], capture_output=True, text=True)
    assert out.returncode == 0
    assert [int(x) for x in out.stdout.split()] == want


def test_failure_is_passed_on(driver):
    out = subprocess.run([driver, "ffe", "1"], capture_output=True, text=True)
    other, rc = (int(x) for x in out.stdout.split()[:2])
    assert other == 0 and rc > 0

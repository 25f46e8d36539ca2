"""The factored-sweep planner (doki_b200/csrc/dk_plan_fx.c) under AddressSanitizer and
UndefinedBehaviorSanitizer, on CPU: the random circuits of test_sanitize_plan (dense,
diagonal, anti-diagonal, phase, sign and X gates on 1 to 5 qubits, 3 to 30 qubits,
every tile width, brickwork layers), and the same with unitary one-qubit gates, whose
factors move from gate to gate.  The driver walks every table of a factored program
and checks that it lies inside the program."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT
from tests.test_sanitize_plan import DRIVER

BUILD = """		dk_plan plan;
		memset(&plan, 0, sizeof(plan));
		const int rc = dk_plan_build(ops, nops, n, prec, &lim, &plan);"""
FREE = "		dk_plan_free(&plan);\n"

WALK = r"""
#include <math.h>
static void unitary(struct dk_gate *g)
{
	const double t = 3 * unit(), p = 6 * unit(), l = 6 * unit();
	double *m = g->m;
	m[0] = cos(t), m[1] = 0;
	m[2] = -cos(l) * sin(t), m[3] = -sin(l) * sin(t);
	m[4] = cos(p) * sin(t), m[5] = sin(p) * sin(t);
	m[6] = cos(p + l) * cos(t), m[7] = sin(p + l) * cos(t);
}

static int check_program(const unsigned char *prog, unsigned n, int prec)
{
	const dk_sweep_hdr *h = (const dk_sweep_hdr *)prog;
	const unsigned amp = prec == DK_C64 ? 8 : 16;
	if (h->mode != DK_SWEEP_FACTORED)
		return h->npass > 0 ? 0 : 1;
	if (h->npass < 1 || h->npass > DK_MAX_FX_PASSES || h->n != (int)n ||
	    h->bytes > DK_FX_BYTES_SMALL || h->ncond > DK_FX_MAX_CONDS)
		return 2;
	const dk_fx_pass *ps = (const dk_fx_pass *)(prog + h->pass_off);
	const dk_fx_list *ls = (const dk_fx_list *)(ps + h->npass);
	const dk_fx_op *os = (const dk_fx_op *)(prog + h->gate_off);
	if ((const unsigned char *)os < (const unsigned char *)ls ||
	    h->gate_off + (unsigned)h->ngate * sizeof(*os) > h->cond_off ||
	    h->cond_off + h->ncond * sizeof(dk_gate_cond) > h->mat_off || h->mat_off > h->bytes)
		return 3;
	const unsigned tile = amp << h->m;
	for (int i = 0; i < h->npass; i++) {
		const dk_fx_pass *p = &ps[i];
		const unsigned nc = p->cond >> 15;
		if (nc > DK_FX_COND || (const void *)(ls + p->list + (1u << nc)) > (const void *)os)
			return 4;
		for (unsigned c = 0; c < nc; c++)
			if ((p->cond >> (5 * c) & 31u) >= h->ncond)
				return 5;
		for (int j = 0; j < 32; j++)
			if (p->slo[j] >= tile || p->rlo[j] >> h->m)
				return 6;
		for (int j = 0; j < 8; j++)
			if (p->shi[j] >= tile || p->rhi[j] >> h->m)
				return 7;
		for (unsigned v = 0; v < 1u << nc; v++) {
			const dk_fx_list *l = &ls[p->list + v];
			if (l->op0 > l->op1 || l->op1 > h->ngate)
				return 8;
			for (int j = 0; j < DK_FX_BITS; j++)
				if (l->gt[j] >= tile || l->st[j] >= tile)
					return 9;
			for (int k = l->op0; k < l->op1; k++) {
				const dk_fx_op *o = &os[k];
				const unsigned z = o->code;
				unsigned b = 0;
				if (z == DK_FX_STAGE)
					b = 64 + (o->mask & 16 ? 16 * amp : 0);
				else if (z < DK_FX_PHASE)
					b = 128;
				else if (z == DK_FX_PHASE)
					b = 16;
				else if (z > DK_FX_NEG)
					return 10;
				if (h->mat_off + 16 * o->coef + b > h->bytes || o->lc >> h->m || o->la >> h->m)
					return 11;
			}
		}
	}
	return 0;
}
"""

STEPS = """		if (t & 1)
			for (int i = 0; i < nops; i++)
				if (ops[i].k == 1 && below(4))
					unitary(gates[i]);
		dk_fx_plan *plan = NULL;
		int rc = dk_fx_begin(ops, nops, n, prec, &lim, &plan);
		long done = 0;
		dk_step step;
		const unsigned char *prog = NULL;
		int bad = 0, more = 0;
		while (rc == 0 && !bad && (more = dk_fx_next(plan, &step, &prog)) > 0) {
			done += step.ngates;
			if (step.kind == 1) {
				/* a copy of its own size: nothing is read past its end */
				const uint32_t bytes = ((const dk_sweep_hdr *)prog)->bytes;
				unsigned char *own = malloc(bytes);
				memcpy(own, prog, bytes);
				bad = check_program(own, n, prec);
				free(own);
			} else if (step.kind != 2 || step.op_index < 0 || step.op_index >= nops) {
				bad = 20;
			}
		}
		if (more < 0 || (!bad && done != nops))
			bad = 21;
"""


def driver_source():
    a = DRIVER.index(BUILD)
    b = DRIVER.index("		const int bad = check_plan(&plan, nops);")
    src = DRIVER[:a] + STEPS + "		if (rc != 0)\n			return 10;\n" + DRIVER[b:]
    src = src.replace("		const int bad = check_plan(&plan, nops);\n", "")
    assert FREE in src
    src = src.replace(FREE, "		dk_fx_end(plan);\n")
    # the plan's checker is not needed; the walk takes its place
    c, d = src.index("static int check_plan("), src.index("int main(")
    return src[:c] + WALK + src[d:]


def test_factored_planner_under_asan_and_ubsan(tmp_path):
    csrc = os.path.join(ROOT, "doki_b200", "csrc")
    drv, exe = tmp_path / "driver.c", tmp_path / "driver"
    drv.write_text(driver_source())
    r = subprocess.run([shutil.which("gcc") or "/usr/bin/gcc", "-std=gnu11", "-O1", "-g",
                        "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
                        "-fno-omit-frame-pointer", "-I", os.path.join(ROOT, "include"), "-I", csrc,
                        "-I", "/usr/local/cuda/include", os.path.join(csrc, "dk_plan.c"),
                        os.path.join(csrc, "dk_plan_fx.c"), str(drv), "-lm", "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0 and "asan" in r.stderr.lower():
        pytest.skip("sanitizer runtime unavailable: " + r.stderr[-200:])
    assert r.returncode == 0, r.stderr
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=1:abort_on_error=0",
               UBSAN_OPTIONS="print_stacktrace=1")
    run = subprocess.run([str(exe), "600"], capture_output=True, text=True, env=env, timeout=900)
    if run.returncode != 0 and "LeakSanitizer has encountered a fatal error" in run.stderr:
        env["ASAN_OPTIONS"] = "detect_leaks=0"
        run = subprocess.run([str(exe), "600"], capture_output=True, text=True, env=env,
                             timeout=900)
    assert run.returncode == 0, run.stdout + run.stderr[-3000:]
    assert run.stdout.strip() == "ok 600"

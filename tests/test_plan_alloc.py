"""Host allocation failures in the factored-sweep planner (doki_b200/csrc/dk_plan_fx.c),
on CPU: a C driver in which allocations fail on demand.  Sweeps change a register in
place while the next ones are planned, so a plan of factored sweeps may fail when it
begins and not later; a plan with other sweeps in it may fail at any step and then
names the gates that are left.  Under AddressSanitizer: nothing is lost or used again on the way."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

DRIVER = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "dk_internal.h"

static long left = -1; /* allocations until all fail, -1: none fails */
static long made;
void *__real_malloc(size_t), *__real_calloc(size_t, size_t), *__real_realloc(void *, size_t);
static int fails(void)
{
	made++;
	if (left < 0)
		return 0;
	return left-- <= 0 ? (left = 0, 1) : 0;
}
void *__wrap_malloc(size_t n) { return fails() ? NULL : __real_malloc(n); }
void *__wrap_calloc(size_t a, size_t b) { return fails() ? NULL : __real_calloc(a, b); }
void *__wrap_realloc(void *p, size_t n) { return fails() ? NULL : __real_realloc(p, n); }

static uint64_t rs = 88172645463325252ull;
static uint64_t rnd(void) { rs ^= rs << 13; rs ^= rs >> 7; rs ^= rs << 17; return rs; }
static unsigned below(unsigned n) { return (unsigned)(rnd() % n); }
static double angle(void) { return (double)(rnd() >> 11) / 9007199254740992.0 * 6.283185307179586; }

static struct dk_gate *make(unsigned k, int kind)
{
	struct dk_gate *g = __real_calloc(1, sizeof(*g));
	g->k = k;
	g->dim = 1ull << k;
	double *m = g->m = __real_calloc(2 * g->dim * g->dim, sizeof(double));
	if (kind == 0) { /* U3 */
		const double t = angle() / 2, p = angle(), l = angle();
		m[0] = cos(t);
		m[2] = -cos(l) * sin(t), m[3] = -sin(l) * sin(t);
		m[4] = cos(p) * sin(t), m[5] = sin(p) * sin(t);
		m[6] = cos(p + l) * cos(t), m[7] = sin(p + l) * cos(t);
	} else if (kind == 1) { /* X */
		m[2] = m[4] = 1;
	} else if (kind == 2) { /* diagonal */
		for (uint64_t e = 0; e < g->dim; e++) {
			const double a = angle();
			m[2 * (e * g->dim + e)] = cos(a), m[2 * (e * g->dim + e) + 1] = sin(a);
		}
	} else { /* dense */
		for (uint64_t e = 0; e < 2 * g->dim * g->dim; e++)
			m[e] = cos(angle());
	}
	return g;
}

static uint64_t support(const dk_flat_op *op)
{
	uint64_t s = op->cm | op->am;
	for (unsigned j = 0; j < op->k; j++)
		s |= 1ull << op->tg[j];
	return s;
}

int main(int argc, char **argv)
{
	const int trials = atoi(argv[1]), dense = atoi(argv[2]);
	long begun = 0, during = 0, refused = 0;
	for (int t = 0; t < trials; t++) {
		const unsigned n = 4 + below(27);
		const int nops = 1 + (int)below(t % 8 == 0 ? 1500 : 200);
		const unsigned few = t % 3 ? n : 4; /* long lists on few qubits */
		dk_flat_op *ops = __real_calloc((size_t)nops, sizeof(*ops));
		struct dk_gate **gates = __real_calloc((size_t)nops, sizeof(*gates));
		for (int i = 0; i < nops; i++) {
			int kind = (int)below(4);
			kind = kind == 3 ? 0 : kind;
			unsigned k = kind == 2 ? 1 + below(3) : 1;
			if (dense && below(12) == 0)
				kind = 3, k = 1 + below(4);
			ops[i].gate = gates[i] = make(k, kind);
			ops[i].k = k;
			uint64_t taken = 0;
			for (unsigned j = 0; j < k; j++) {
				unsigned q;
				do
					q = below(few);
				while (taken >> q & 1);
				taken |= 1ull << q;
				ops[i].tg[j] = q;
			}
			for (unsigned c = below(4); c && (unsigned)__builtin_popcountll(taken) < n; c--) {
				unsigned q;
				do
					q = below(n);
				while (taken >> q & 1);
				taken |= 1ull << q;
				*(below(2) ? &ops[i].cm : &ops[i].am) |= 1ull << q;
			}
		}
		const int prec = below(2) ? DK_C128 : DK_C64;
		dk_plan_limits lim;
		memset(&lim, 0, sizeof(lim));
		lim.tile_bits = below(3) ? 0 : 4 + (int)below(9);
		dk_plan_default_limits(prec, n, &lim);
		dk_fx_plan *p = NULL;
		/* every allocation of the beginning in turn */
		int rc = DK_ERR_ALLOC;
		for (long k = 0; rc == DK_ERR_ALLOC && k < 100; k++) {
			left = k;
			rc = dk_fx_begin(ops, nops, n, prec, &lim, &p);
			if (rc == 0 && dk_fx_all(p) && (rc = dk_fx_reserve(p)) != 0)
				dk_fx_end(p);
			left = -1;
			begun++;
		}
		if (rc)
			return 2;
		const int all = dk_fx_all(p);
		if (!dense && !all)
			return 3;
		long gates_done = 0;
		dk_step step;
		const unsigned char *prog;
		if (all) {
			left = 0;
			const long before = made;
			while ((rc = dk_fx_next(p, &step, &prog)) > 0)
				gates_done += step.ngates;
			left = -1;
			during += made - before;
			if (rc || gates_done != nops) {
				printf("trial %d: %d, %ld of %d gates\n", t, rc, gates_done, nops);
				return 4;
			}
		} else {
			const int reserved = below(4) != 0;
			if (reserved && dk_fx_reserve(p))
				return 12;
			left = (long)below(60);
			while ((rc = dk_fx_next(p, &step, &prog)) > 0)
				gates_done += step.kind == 1 ? step.ngates : 1;
			left = -1;
			if (rc != 0 && rc != -DK_ERR_ALLOC)
				return 5;
			refused += rc != 0;
			/* what is left after a failure: every gate that no step holds, after
			 * all gates before it that it depends on */
			int *ids = __real_calloc((size_t)nops, sizeof(int));
			char *in = __real_calloc((size_t)nops, 1);
			const int rest = rc && reserved ? dk_fx_left(p, ids) : 0;
			if (rest < 0 || ((!rc || reserved) && gates_done + rest != nops))
				return 6;
			for (int i = 0; i < rest; i++) {
				if (ids[i] < 0 || ids[i] >= nops || in[ids[i]]++)
					return 7;
				const uint64_t si = support(&ops[ids[i]]);
				for (int j = 0; j < i; j++)
					if (ids[j] > ids[i] && support(&ops[ids[j]]) & si)
						return 8;
			}
			for (int i = 0; i < rest; i++)
				for (int j = ids[i] + 1; j < nops; j++)
					if (rest && !in[j] && support(&ops[j]) & support(&ops[ids[i]]))
						return 9; /* j ran before a gate that it comes after */
			free(ids);
			free(in);
		}
		dk_fx_end(p);
		for (int i = 0; i < nops; i++) {
			free(gates[i]->m);
			free(gates[i]);
		}
		free(gates);
		free(ops);
	}
	printf("%ld %ld %ld\n", begun, during, refused);
	return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("plan_alloc")
    csrc = os.path.join(ROOT, "doki_b200", "csrc")
    src, exe = tmp / "driver.c", tmp / "driver"
    src.write_text(DRIVER)
    r = subprocess.run([shutil.which("gcc") or "/usr/bin/gcc", "-std=gnu11", "-O1", "-g",
                        "-fsanitize=address", "-fno-omit-frame-pointer",
                        "-Wl,--wrap=malloc,--wrap=calloc,--wrap=realloc",
                        "-I", os.path.join(ROOT, "include"), "-I", csrc,
                        "-I", "/usr/local/cuda/include", os.path.join(csrc, "dk_plan.c"),
                        os.path.join(csrc, "dk_plan_fx.c"), str(src), "-lm", "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0 and "asan" in r.stderr.lower():
        pytest.skip("sanitizer runtime unavailable: " + r.stderr[-200:])
    assert r.returncode == 0, r.stderr
    return str(exe)


def run(driver, *args):
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=1:allocator_may_return_null=1")
    r = subprocess.run([driver, *args], capture_output=True, text=True, env=env, timeout=600)
    if r.returncode != 0 and "LeakSanitizer has encountered a fatal error" in r.stderr:
        env["ASAN_OPTIONS"] = "detect_leaks=0:allocator_may_return_null=1"
        r = subprocess.run([driver, *args], capture_output=True, text=True, env=env, timeout=600)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-3000:])
    return [int(x) for x in r.stdout.split()]


def test_factored_plans_allocate_at_the_beginning_only(driver):
    begun, during, _ = run(driver, "250", "0")
    assert begun > 10 * 250  # each of a beginning's allocations failed once
    assert during == 0


def test_other_plans_fail_with_a_status(driver):
    _, during, refused = run(driver, "250", "1")
    assert during == 0 and refused > 20

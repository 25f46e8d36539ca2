"""The ring that programs and matrices of a flush pass through on their way to the
device (doki_b200/csrc/dk_stage_ring.h), on CPU: a driver in which a copy to the
device runs only when the host waits for an event recorded behind it.  No byte may
be written again before its copy has run."""
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
#include <vector>
#include "dk_stage_ring.h"

constexpr size_t PART = 1u << 20;
struct Copy { size_t at, bytes; };

int main(int argc, char **argv)
{
	/* sizes: argv[1] a list, or argv[1] = "random" and a seed */
	std::vector<size_t> sizes;
	if (!strcmp(argv[1], "random")) {
		unsigned long long x = 88172645463325252ull + strtoull(argv[2], 0, 10) * 7919;
		for (int i = 0; i < 20000; ++i) {
			x ^= x << 13; x ^= x >> 7; x ^= x << 17;
			const int k = (int)(x % 7);
			sizes.push_back(k < 4 ? 64 + (x >> 8) % (40u << 10)
					: k == 4 ? (size_t)256 << ((x >> 8) % 13) /* to 1 MiB */
					: k == 5 ? 16 + (x >> 8) % PART : PART - 256 * ((x >> 8) % 4));
		}
	} else {
		const size_t n = strtoull(argv[1], 0, 10), count = strtoull(argv[2], 0, 10);
		sizes.assign(count, n);
	}
	dk::StageRing<PART, 2> ring;
	std::vector<Copy> queued; /* in stream order, not yet run */
	size_t done = 0, mark[2] = { 0, 0 }; /* copies run; stream length at an event */
	size_t waits = 0, depth = 0;
	for (size_t bytes : sizes) {
		size_t at = ~(size_t)0;
		const int rc = ring.place(
			bytes, [&](int p) { mark[p] = queued.size(); return 0; },
			[&](int p) { if (mark[p] > done) done = mark[p]; ++waits; return 0; }, &at);
		if (rc || at % 256 || at + bytes > 2 * PART || at / PART != (at + bytes - 1) / PART)
			return 2;
		for (size_t i = done; i < queued.size(); ++i)
			if (at < queued[i].at + queued[i].bytes && queued[i].at < at + bytes) {
				printf("%zu bytes at %zu written over a queued copy\n", bytes, at);
				return 1;
			}
		queued.push_back({ at, bytes });
		if (queued.size() - done > depth)
			depth = queued.size() - done;
	}
	printf("ok %zu %zu\n", waits, depth);
	return 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("ring")
    src, exe = tmp / "driver.cpp", tmp / "driver"
    src.write_text(DRIVER)
    r = subprocess.run([shutil.which("g++") or "/usr/bin/g++", "-std=c++17", "-O1",
                        "-I", os.path.join(ROOT, "doki_b200", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(exe)


@pytest.mark.parametrize("qubits", range(1, 9))
def test_matrices_that_divide_a_part(driver, qubits):
    """Matrices of gates on 1 to 8 qubits (16 x 4^k bytes; 8: a whole part): a part
    that is exactly full."""
    size = 16 * 4 ** qubits
    count = 4 * ((1 << 20) // max(size, 256)) + 3
    out = subprocess.run([driver, str(size), str(count)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_random_sizes(driver):
    for seed in range(20):
        out = subprocess.run([driver, "random", str(seed)], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout
        waits, depth = (int(x) for x in out.stdout.split()[1:])
        assert waits > 100 and depth > 10  # parts change, copies stay queued


def test_failures_leave_the_place(tmp_path):
    src, exe = tmp_path / "f.cpp", tmp_path / "f"
    src.write_text(r"""
#include "dk_stage_ring.h"
int main()
{
	dk::StageRing<1024, 2> r;
	size_t at = 7;
	auto ok = [](int) { return 0; };
	auto bad = [](int) { return 5; };
	if (r.place(1024, ok, ok, &at) || at != 0)
		return 1;
	if (r.place(16, bad, ok, &at) != 5 || r.part != 0 || at != 0)
		return 2;
	if (r.place(1024, ok, bad, &at) || at != 1024) /* part 1 was never left: no wait */
		return 3;
	if (r.place(16, ok, bad, &at) != 5 || r.part != 1)
		return 4;
	return r.place(16, ok, ok, &at) || at != 0;
}
""")
    r = subprocess.run([shutil.which("g++") or "/usr/bin/g++", "-std=c++17", "-I",
                        os.path.join(ROOT, "doki_b200", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(exe)]).returncode == 0

"""What the factored-sweep planner leaves of a one-qubit matrix, on CPU: the matrix
that a plan applies, against the one that was given."""
from __future__ import annotations

import numpy as np
import pytest

from doki_b200 import workloads as W
from tests.test_plan import HDR, lib, replay_sweep  # noqa: F401
from tests.test_plan_factored import plan, replay


def applied(lib, m):  # noqa: F811
    """The matrix that the plan of one gate applies, and the kind of its sweep."""
    (_, blob, _, _), = plan(lib, [W.Op(m, [0])], 4)
    mode = int(np.frombuffer(blob, HDR, 1)[0]["mode"])
    cols = []
    for j in (0, 1):
        psi = np.zeros(16, dtype=np.complex128)
        psi[j] = 1
        cols.append((replay(blob, psi, 2) if mode == 2 else replay_sweep(blob, 0, psi))[:2])
    return np.array(cols).T, mode


# A factoring holds 7 of a matrix's 8 real numbers.  The phase of b c / (a d) that it
# leaves out is at most 4e-15 next to entries of size 1, else the matrix is applied as
# it was given; a quarter of it goes to each entry (a half to b and c where they are
# small).  The factors and their products add five roundings of 2^-53 each.
BOUND = 4e-15 / 2 + 5 * 2.0 ** -53


@pytest.mark.parametrize("defect", [0.0, 1e-15, 3e-15, 5e-15, 7e-15])
def test_matrices_a_little_off_unitary(lib, defect):  # noqa: F811
    """A phase on one entry: within the 1e-14 that counts as unitary."""
    modes = set()
    for seed in range(60):
        rng = W.rng_for(8400 + seed)
        m = W.u3(*rng.uniform(0, 6, 3))
        m[tuple(rng.integers(0, 2, 2))] *= np.exp(1j * defect * rng.choice([-1, 1]))
        got, mode = applied(lib, m)
        modes.add(mode)
        assert np.max(np.abs(got - m)) < BOUND, (seed, mode)
    if defect == 0.0:
        assert modes == {2}


def test_small_and_large_angles(lib):  # noqa: F811
    """Entries of very different size keep their own accuracy: the phase left out of
    a small entry is a small part of it."""
    for theta in (1e-3, 1e-7, 1e-12, np.pi - 1e-3, np.pi - 1e-7):
        for seed in range(20):
            rng = W.rng_for(8500 + seed)
            m = W.u3(theta, *rng.uniform(0, 6, 2))
            got, mode = applied(lib, m)
            assert mode == 2
            assert (np.abs(got - m) <= BOUND * np.abs(m)).all()


def test_quarter_of_the_phase(lib):  # noqa: F811
    """Where all four entries are alike, each takes a quarter of what is left out:
    with 3.2e-15 of it, 0.8e-15 and the roundings."""
    for seed in range(40):
        rng = W.rng_for(8600 + seed)
        m = W.u3(np.pi / 2 + 0.1 * rng.random(), *rng.uniform(0, 1, 2))
        m[0, 1] *= 1 + 2.2e-15j
        got, mode = applied(lib, m)
        if mode == 2:
            assert np.max(np.abs(got - m)) < 3.2e-15 / 4 + 5 * 2.0 ** -53

"""When a job's refinement stops (lsms_b200/csrc/refine_rule.h): the rule itself on the host, and jobs that
need it on the GPU."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

from lsms_b200 import tau as T
from lsms_b200 import workloads as W

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lsms_b200", "csrc")
CONVERGED, DIVERGED = 1, 2


@pytest.fixture(scope="module")
def state(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text('#include "refine_rule.h"\n'
                                'extern "C" int state(double c, double p, double p2, int acc, int last) '
                                '{ return b200::refine_state(c, p, p2, acc != 0, last != 0); }\n')
    so = str(d / "rule.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "rule.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).state
    f.argtypes = [ctypes.c_double] * 3 + [ctypes.c_int] * 2
    return f


def _run(state, sizes, accelerated, rounds=10):
    """(round that stopped, state) of a job with these correction sizes."""
    p = p2 = 0.0
    for i, c in enumerate(sizes, 1):
        s = state(c, p, p2, accelerated, i == rounds)
        if s:
            return i, s
        p, p2 = c, p
    return None


@pytest.mark.parametrize("sizes,want", [
    # a large drop says nothing about the next rounds: the next correction stalls, or grows, far above the floor
    ([1e-4, 1e-8, 2e-8], None),
    ([1e-4, 1e-8, 1e-5], (3, DIVERGED)),
    ([1e-2, 1.1e-4, 3.8e-9], None),
    ([1e-2, 1.1e-4, 3.8e-9, 4.7e-11, 1e-13], (5, CONVERGED)),
    # the first two corrections are those of plain rounds
    ([1e-4, 1e-10], (2, CONVERGED)),
    ([1e-6, 1e-8, 1e-10, 1e-12], (4, CONVERGED)),
    # a stalled job at its rounding floor, and one above it
    ([1e-3, 1e-4, 8e-5, 5e-13, 6e-13], (5, CONVERGED)),
    ([1e-3, 1e-4, 8e-5, 2e-12, 3e-12], None),
    # the last of ten rounds
    ([1e-3 * 0.3 ** i for i in range(9)] + [1e-8], None),
    ([1e-3 * 0.3 ** i for i in range(9)] + [9e-13], (10, CONVERGED)),
    ([np.nan], (1, DIVERGED)),
    ([1e-4, np.inf], (2, DIVERGED)),
])
def test_accelerated_rounds(state, sizes, want):
    assert _run(state, sizes, True) == want


@pytest.mark.parametrize("sizes,want", [
    ([1e-4, 1e-8], (2, CONVERGED)),
    ([1e-4, 1e-7, 1e-7], (3, DIVERGED)),
    ([1e-4, 1e-7, 0.99e-10], (3, CONVERGED)),
    ([9e-13], (1, CONVERGED)),
    ([2e-12, 2e-12], (2, DIVERGED)),
    ([np.nan], (1, DIVERGED)),
])
def test_plain_rounds(state, sizes, want):
    assert _run(state, sizes, False) == want


@pytest.mark.gpu
def test_poor_factors_are_refined_far_enough():
    """Jobs of the non-collinear batch (N = 4320) whose accelerated corrections fall by 3e-5 in one round and
    by a hundred in the next.  The FP64 results are within 3e-13 of 64-bit arithmetic, and a converged job's
    estimated error is below 1e-12."""
    wl = W.config_noncollinear_batch(seed=3)
    s = T.TauSolver(wl.lmax, wl.n_spin_cant, wl.n_spin_pola)
    try:
        s.upload_tmat(wl.tmat_store)
        specs = []
        for k, (atom, iie) in enumerate([(45, 9), (62, 10), (24, 1)]):
            at = wl.atoms[atom]
            s.set_atom(k, at.liz_pos, at.liz_lmax, at.liz_store_idx, at.ubr, at.ubrd)
            specs.append((k, iie, 0, wl.energies[iie]))
        want = s.solve_jobs(T.make_jobs(specs), T.PREC_FP64)
        got = s.solve_jobs(T.make_jobs(specs), T.PREC_MIXED)
    finally:
        s.close()
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= 1e-11 * np.abs(w).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [100, 240])
def test_values_past_fp32_are_solved_in_fp64(solver_factory, n):
    """A matrix whose inverse does not fit FP32 factors: the refinement's NaN does not count as converged."""
    rng = np.random.default_rng(n)
    m = 1e-40 * (np.eye(n) + 0.4 / np.sqrt(n) * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))))
    t0 = rng.normal(size=(16, 16)) + 1j * rng.normal(size=(16, 16))
    rhs = np.zeros((n, 16), np.complex128)
    rhs[:16] = t0
    want = np.linalg.solve(m, rhs)[:16]
    got = solver_factory(3, 1, 1).solve_tau00_dense(m, t0, T.PREC_MIXED)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()

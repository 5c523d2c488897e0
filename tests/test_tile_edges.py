"""Edges of the kernels' tiles: sizes at which a tile, a block or an aligned copy ends inside a row."""

import numpy as np
import pytest

from lsms_b200 import tau as T
from lsms_b200 import workloads as W

TOL_MIXED = 1e-10


def _lmax_step_problem(lattice, shells, n_reduced, seed):
    """The outer n_reduced sites at lmax 2 (blocks of 9)."""
    a = {"bcc": 5.42, "fcc": 6.82}[lattice]
    L = W.lattice_shells(lattice, a, shells).shape[1]
    lmax = np.full(L, 3, np.int32)
    lmax[L - n_reduced:] = 2
    return W.make_problem(lattice, a, shells, 3, [0.5 + 0.1j, -0.1 + 0.3j], seed, n_species=2, liz_lmax=lmax)


def _tau_err(prob, iie, got):
    from oracle import port
    want = port.solve(prob, iie)
    t0 = -port.tau00_l(prob, np.zeros((prob.kkrsz_ns, prob.kkrsz_ns), np.complex128), iie)
    return np.abs(got - want).max() / np.abs(want + t0).max()


@pytest.mark.gpu
@pytest.mark.parametrize("pivoting", [T.PIVOT_BLOCK, T.PIVOT_PANEL])
@pytest.mark.parametrize("lattice,shells,n_reduced", [("bcc", 2, 7), ("bcc", 2, 1), ("fcc", 3, 21), ("fcc", 4, 5)])
def test_mixed_odd_size(solver_factory, lattice, shells, n_reduced, pivoting):
    """An odd n puts the trailing block of the last step on an odd row: the tensor-core update's
    16-byte-aligned reduce-add cannot start there."""
    prob = _lmax_step_problem(lattice, shells, n_reduced, 21)
    assert (prob.nrmat_ns - 16) % 2 == 1
    s = solver_factory(3, 1, 1)
    s.load_problem(prob)
    s.set_pivoting(pivoting)
    try:
        out = s.solve_jobs(T.make_jobs([(0, i, 0, e) for i, e in enumerate(prob.energies)]), T.PREC_MIXED)
        assert s.last_fallback_count == 0
    finally:
        s.set_pivoting(T.PIVOT_AUTO)
    for i in range(2):
        assert _tau_err(prob, i, out[i]) <= TOL_MIXED

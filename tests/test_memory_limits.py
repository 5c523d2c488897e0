"""FP64 waves when device memory is nearly used up: the digit planes of the integer tensor-core update."""

import numpy as np
import pytest

from lsms_b200 import tau as T
from lsms_b200 import workloads as W

MB = 1 << 20


def _hog(leave):
    """Device memory held so that about `leave` bytes are free."""
    import torch
    held = []
    for _ in range(3):
        n = torch.cuda.mem_get_info()[0] - int(leave)
        if n < 4 * MB:
            break
        held.append(torch.empty(n // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda"))
    return held


def _release(held):
    import torch
    held.clear()
    torch.cuda.empty_cache()


class _Waves:
    """One solver with an atom of each number of shells; batches of `n` energies of one of them."""

    def __init__(self, shells, n):
        self.energies = W.semicircle_contour(-0.2, 0.7, n)
        prob = W.make_problem("fcc", 6.82, shells[0], 3, self.energies, 3, n_species=2)
        self.s = T.TauSolver(3, 1, 1)
        self.s.upload_tmat(prob.tmat_store)
        for i, sh in enumerate(shells):
            p = W.make_problem("fcc", 6.82, sh, 3, self.energies, 3, n_species=2)
            self.s.set_atom(sh, p.liz_pos, p.liz_lmax, np.minimum(p.liz_store_idx, 1), p.ubr, p.ubrd)

    def solve(self, shells, n):
        out = self.s.solve_jobs(T.make_jobs([(shells, i, 0, self.energies[i]) for i in range(n)]), T.PREC_FP64)
        return out, self.s.last_launch_count


def _close(a, b):
    return np.abs(a - b).max() <= 1e-10 * np.abs(b).max()


@pytest.mark.gpu
def test_planes_that_find_no_room():
    """A wave whose planes do not fit runs without them, and a smaller one still uses the planes it had."""
    w = _Waves((2, 5), 16)  # N = 304, 1264
    try:
        want_big = w.solve(5, 8)[0]
        want, launches = w.solve(5, 4)
    finally:
        w.s.close()
    w = _Waves((2, 5), 16)
    held = []
    try:
        first, count = w.solve(5, 4)  # planes for four slots
        assert count == launches
        w.solve(2, 16)                # sixteen slots, but updates too small for planes
        held = _hog(32 * MB)          # the planes of sixteen slots take 63 MB
        for _ in range(3):
            assert _close(w.solve(5, 8)[0], want_big)
        again, count = w.solve(5, 4)
        assert count == launches      # (a wave on the FP64 tensor cores alone takes fewer launches)
        assert np.array_equal(again, want) and np.array_equal(first, want)
        _release(held)
        got, _ = w.solve(5, 8)
        assert np.array_equal(got, want_big)
    finally:
        w.s.close()
        _release(held)


@pytest.mark.gpu
def test_waves_do_not_depend_on_the_planes_held():
    """The same call twice with little memory: the planes allocated by the first count as available to the
    second, so both take the same waves."""
    w = _Waves((6,), 16)
    held = []
    try:
        w.solve(6, 1)  # what a context allocates besides the wave's slots
        ld = 1408
        planes = ld * (3 * 8 * 128 + 16) + 256
        slot = 32 * ld * ld + 3 * ld * 32 * 16 + planes
        held = _hog(2 * 6.16 * slot - 32 * ld * ld - planes)  # six slots and a sixth (one is held)
        counts = [w.solve(6, 16)[1] for _ in range(3)]
        assert len(set(counts)) == 1
    finally:
        w.s.close()
        _release(held)

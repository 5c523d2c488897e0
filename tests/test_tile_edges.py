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


def _dense(n, b, seed, shuffle=False):
    """A well-conditioned complex matrix (condition number of a few tens at most) and a t0; with
    `shuffle` its rows past the central block are permuted, so that pivots leave the diagonal blocks."""
    rng = np.random.default_rng(seed)
    m = np.eye(n) + 0.4 / np.sqrt(n) * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
    if shuffle:
        m[b:] = m[b + rng.permutation(n - b)]
    t0 = rng.normal(size=(b, b)) + 1j * rng.normal(size=(b, b))
    rhs = np.zeros((n, b), np.complex128)
    rhs[:b] = t0
    return m, t0, np.linalg.solve(m, rhs)[:b]


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(T.PREC_FP64, 1e-12), (T.PREC_MIXED, TOL_MIXED)])
@pytest.mark.parametrize("b", [1, 9, 16, 32])
@pytest.mark.parametrize("rest", [0, 1, 15, 17, 63, 64, 65, 80, 129, 193, 447])
def test_dense_edge_sizes(solver_factory, prec, tol, b, rest):
    """n = b + rest around the 64-column steps, the 16- and 64-row tiles and the 8-wide fragments."""
    m, t0, want = _dense(b + rest, b, 100 * b + rest)
    got = solver_factory(3, 1, 1).solve_tau00_dense(m, t0, prec)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(T.PREC_FP64, 1e-12), (T.PREC_MIXED, TOL_MIXED)])
@pytest.mark.parametrize("rest", [70, 191, 321, 700])
def test_dense_panel_pivoting(solver_factory, prec, tol, rest):
    """Rows in random order: every step's pivots come from below its diagonal block, with the candidates
    filtered once more than 256 rows are left."""
    m, t0, want = _dense(16 + rest, 16, rest, shuffle=True)
    s = solver_factory(3, 1, 1)
    s.set_pivoting(T.PIVOT_PANEL)
    try:
        got = s.solve_tau00_dense(m, t0, prec)
    finally:
        s.set_pivoting(T.PIVOT_AUTO)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,shells,n_reduced", [("bcc", 1, 3), ("bcc", 3, 4), ("fcc", 3, 20)])
def test_full_tau_and_adjoint_odd_sizes(solver_factory, lattice, shells, n_reduced):
    """The inverse's tiles at sizes that are no multiple of 16: tau over the LIZ, and the gradients from
    the dense inverse."""
    from oracle import port
    prob = _lmax_step_problem(lattice, shells, n_reduced, 8)
    s = solver_factory(3, 1, 1)
    s.load_problem(prob)
    n, e = prob.nrmat_ns, prob.energies[0]
    m = port.build_kkr(prob, 0)
    off = np.concatenate([[0], np.cumsum((prob.liz_lmax + 1) ** 2)])
    t = [prob.t_block(int(i), 0)[:k, :k] for i, k in zip(prob.liz_store_idx, np.diff(off))]
    inv = np.linalg.inv(m)
    want = np.concatenate([inv[:, off[j]:off[j + 1]] @ t[j] for j in range(len(t))], axis=1)
    got = s.solve_tau_full(0, 0, 0, e, n)
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
    rng = np.random.default_rng(2)
    bar = rng.normal(size=(16, 16)) + 1j * rng.normal(size=(16, 16))
    _, tbar, dlog = s.solve_vjp(T.make_jobs([(0, 0, 0, e)]), bar[None], [prob.num_liz])
    g = np.concatenate([np.linalg.solve(t[j], (np.eye(n) - m)[off[j]:off[j + 1]]) for j in range(len(t))])
    z, h, lam = g @ (inv[:, :16] @ t[0]), g @ inv, inv[:16].T @ bar
    scale = max(np.abs(lam).max() * np.abs(z).max(), 1.0)
    for j in range(len(t)):
        r, k = slice(off[j], off[j + 1]), off[j + 1] - off[j]
        wb = lam[r] @ z[r].T + (lam[r] if j == 0 else 0.0)
        assert np.abs(tbar[0][j][:k, :k] - wb).max() <= 1e-10 * scale
        assert np.abs(dlog[0][j][:k, :k] + h[r, r].T).max() <= 1e-10 * max(1.0, np.abs(h).max())


@pytest.mark.gpu
@pytest.mark.parametrize("sweep", [T.SWEEP_FP32, T.SWEEP_FP64])
@pytest.mark.parametrize("cant", [1, 2])
@pytest.mark.parametrize("njobs", [1, 2, 7, 33])
def test_batch_sizes(solver_factory, njobs, cant, sweep):
    """Cluster sizes of the sweeps and the residual's split of K follow the number of jobs: each job of a
    batch against the oracle, FP64 and mixed."""
    from oracle import port
    prob = W.make_problem("bcc", 5.42, 2, 3, W.semicircle_contour(-0.2, 0.7, njobs), 5, n_species=None,
                          n_spin_cant=cant, n_spin_pola=cant)
    s = solver_factory(3, cant, cant)
    s.load_problem(prob)
    jobs = T.make_jobs([(0, i, 0, e) for i, e in enumerate(prob.energies)])
    s.set_mixed_sweep(sweep)
    try:
        out = {prec: s.solve_jobs(jobs, prec) for prec in (T.PREC_FP64, T.PREC_MIXED)}
    finally:
        s.set_mixed_sweep(T.SWEEP_FP32)
    for i in range(0, njobs, max(1, njobs // 4)):
        # two backward-stable FP64 solves differ by a few times cond(M) 2^-53 (cond up to 1e4 here)
        bound = max(1e-12, 8 * np.linalg.cond(port.build_kkr(prob, i)) * 2.0 ** -53)
        assert _tau_err(prob, i, out[T.PREC_FP64][i]) <= bound
        assert _tau_err(prob, i, out[T.PREC_MIXED][i]) <= TOL_MIXED


@pytest.mark.gpu
@pytest.mark.parametrize("outer", [3, 2, 1])
@pytest.mark.parametrize("coupled", [False, True])
def test_build_non_collinear_t(solver_factory, outer, coupled):
    """M of a non-collinear t whose spin blocks are diagonal (one product per element), and of one with
    elements off those diagonals, equal lmax and lmax steps."""
    from oracle import port
    L = W.lattice_shells("bcc", 5.42, 1).shape[1]
    lmax = np.full(L, 3, np.int32)
    lmax[L // 2:] = outer
    prob = W.make_problem("bcc", 5.42, 1, 3, [0.4 + 0.2j], 3, n_species=None, n_spin_cant=2, n_spin_pola=2, liz_lmax=lmax)
    if coupled:
        rng = np.random.default_rng(1)
        prob.tmat_store[2:5, 0, :1024] += 0.01 * (rng.normal(size=(3, 1024)) + 1j * rng.normal(size=(3, 1024)))
    s = solver_factory(3, 2, 2)
    s.load_problem(prob)
    got = s.build_kkr(0, 0, 0, prob.energies[0], prob.nrmat_ns)
    want = port.build_kkr(prob, 0)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()

@pytest.mark.gpu
@pytest.mark.parametrize("n_reduced", [0, 3, 10])
def test_updates_by_digit_products(solver_factory, n_reduced):
    """32 jobs of N = 816 and less: the steps with enough rows run on the integer tensor cores, their
    row panels, column tiles and the first block that the look-ahead takes out ending anywhere.  Against
    the oracle, in the batch and alone; the gradients likewise (the inverse's two passes)."""
    from oracle import port
    njobs = 32
    L = W.lattice_shells("bcc", 5.42, 4).shape[1]
    lmax = np.full(L, 3, np.int32)
    lmax[L - n_reduced:] = 2
    prob = W.make_problem("bcc", 5.42, 4, 3, W.semicircle_contour(-0.2, 0.7, njobs), 13, n_species=2, liz_lmax=lmax)
    s = solver_factory(3, 1, 1)
    s.load_problem(prob)
    specs = [(0, i, 0, e) for i, e in enumerate(prob.energies)]
    out = s.solve_jobs(T.make_jobs(specs), T.PREC_FP64)
    rng = np.random.default_rng(2)
    bar = rng.normal(size=(njobs, 16, 16)) + 1j * rng.normal(size=(njobs, 16, 16))
    _, tb, ld = s.solve_vjp(T.make_jobs(specs), bar, [prob.num_liz] * njobs)
    for i in (0, 15, 31):
        # two backward-stable FP64 solves differ by a few times cond(M) 2^-53
        bound = max(1e-12, 8 * np.linalg.cond(port.build_kkr(prob, i)) * 2.0 ** -53)
        assert _tau_err(prob, i, out[i]) <= bound
        alone = s.solve_jobs(T.make_jobs(specs[i:i + 1]), T.PREC_FP64)
        assert _tau_err(prob, i, alone[0]) <= bound
        # the gradients too go through one refined solve
        _, tb1, ld1 = s.solve_vjp(T.make_jobs(specs[i:i + 1]), bar[i:i + 1], [prob.num_liz])
        assert np.abs(tb[i] - tb1[0]).max() <= 10 * bound * np.abs(tb1[0]).max()
        # d ln det M comes from the unrefined inverse, whose error is that of the block LU (pivots inside
        # the diagonal blocks): up to 9 times cond(M) 2^-53 here, by digits as by FP64 products.  Against
        # -((G M^-1)_jj)^T with t_j (G M^-1)_jj = (M^-1 - 1)_jj.
        inv = np.linalg.inv(port.build_kkr(prob, i))
        off = np.concatenate([[0], np.cumsum((lmax + 1) ** 2)])
        err = [0.0, 0.0]
        for j in range(prob.num_liz):
            k = off[j + 1] - off[j]
            t = prob.t_block(int(prob.liz_store_idx[j]), i)[:k, :k]
            want = -np.linalg.solve(t, inv[off[j]:off[j + 1], off[j]:off[j + 1]] - np.eye(k)).T
            err = [max(e, np.abs(d[j][:k, :k] - want).max()) for e, d in zip(err, (ld[i], ld1[0]))]
        assert err[0] <= 8 * err[1] + 10 * bound * np.abs(ld1[0]).max()
        assert err[0] <= 32 * np.linalg.cond(port.build_kkr(prob, i)) * 2.0 ** -53 * np.abs(ld1[0]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,shells,njobs", [("bcc", 2, 1), ("fcc", 3, 1), ("fcc", 7, 1), ("fcc", 7, 2), ("bcc", 2, 65)])
def test_fp64_resolve_job_counts(solver_factory, lattice, shells, njobs):
    """One round converges no job, so every one is re-solved by FP64 block LU, whose update kernel takes
    the wave's tiles on a small looping grid: a wave of one job (alone, or the last one of 65), and of two."""
    from oracle import port
    a = {"bcc": 5.42, "fcc": 6.82}[lattice]
    prob = W.make_problem(lattice, a, shells, 3, W.semicircle_contour(-0.3, 0.7, njobs) if njobs > 1 else [0.35 + 0.15j],
                          31, n_species=2)
    s = solver_factory(3, 1, 1)
    s.load_problem(prob)
    jobs = T.make_jobs([(0, i, 0, e) for i, e in enumerate(prob.energies)])
    want = s.solve_jobs(jobs, T.PREC_FP64)
    s.set_refinement(T.PREC_MIXED, 1)
    try:
        got = s.solve_jobs(jobs, T.PREC_MIXED)
        assert s.last_fallback_count == njobs
    finally:
        s.set_refinement(T.PREC_MIXED, 10)
    for i in range(njobs):
        t0 = -port.tau00_l(prob, np.zeros((16, 16), np.complex128), i)
        assert np.abs(got[i] - want[i]).max() <= 1e-12 * np.abs(want[i] + t0).max()


def _register(s, shells, energies, cant=1, seed=17):
    """Atoms 0, 1, ... with these numbers of fcc shells over one t-matrix store."""
    probs = [W.make_problem("fcc", 6.82, sh, 3, energies, seed, n_species=2, n_spin_cant=cant, n_spin_pola=cant)
             for sh in shells]
    s.upload_tmat(probs[0].tmat_store)
    for a, p in enumerate(probs):
        p.tmat_store, p.liz_store_idx = probs[0].tmat_store, np.minimum(p.liz_store_idx, 1)
        s.set_atom(a, p.liz_pos, p.liz_lmax, p.liz_store_idx, p.ubr, p.ubrd)
    return probs


@pytest.mark.gpu
@pytest.mark.parametrize("shells,cant,nen,pivoting", [
    ((2,), 1, 40, T.PIVOT_BLOCK),           # N = 304: the residual's split
    ((7,), 1, 5, T.PIVOT_BLOCK),            # N = 2160, 688: digit products and FP64 tensor cores
    ((3,), 1, 33, T.PIVOT_BLOCK),
    ((5, 6, 3, 4), 1, 5, T.PIVOT_BLOCK),    # N = 1264, 1392, 688, 880 in one wave
    ((5, 6, 3), 1, 3, T.PIVOT_PANEL),       # row moves between digit products
    ((3, 2), 2, 4, T.PIVOT_BLOCK),          # b = 32, N = 1376 and 608
])
def test_fp64_results_do_not_depend_on_the_batch(solver_factory, shells, cant, nen, pivoting):
    """Every job of a batch, bit for bit the result of the job alone, and against the oracle."""
    from oracle import port
    s = solver_factory(3, cant, cant)
    energies = W.semicircle_contour(-0.2, 0.7, nen)
    probs = _register(s, shells, energies, cant)
    specs = [(a, i, 0, e) for i, e in enumerate(energies) for a in range(len(shells))]
    s.set_pivoting(pivoting)
    try:
        out = s.solve_jobs(T.make_jobs(specs), T.PREC_FP64)
        for j, spec in enumerate(specs):
            assert np.array_equal(out[j], s.solve_jobs(T.make_jobs([spec]), T.PREC_FP64)[0])
    finally:
        s.set_pivoting(T.PIVOT_AUTO)
    for a in range(len(shells) if len(shells) > 1 else 0):
        bound = max(1e-12, 8 * np.linalg.cond(port.build_kkr(probs[a], 1)) * 2.0 ** -53)
        assert _tau_err(probs[a], 1, out[len(shells) + a]) <= bound


@pytest.mark.gpu
def test_gradients_do_not_depend_on_the_batch(solver_factory):
    """The inverse's passes on both sides of the digit products' line, uneven sizes in one wave."""
    s = solver_factory(3, 1, 1)
    energies = W.semicircle_contour(-0.2, 0.7, 3)
    probs = _register(s, (3, 6, 5), energies)
    specs = [(a, i, 0, e) for i, e in enumerate(energies) for a in range(3)]
    num = [probs[a].num_liz for a, _, _, _ in specs]
    rng = np.random.default_rng(4)
    bar = rng.normal(size=(9, 16, 16)) + 1j * rng.normal(size=(9, 16, 16))
    tau, tb, dl = s.solve_vjp(T.make_jobs(specs), bar, num)
    for j, spec in enumerate(specs):
        t1, tb1, dl1 = s.solve_vjp(T.make_jobs([spec]), bar[j:j + 1], num[j:j + 1])
        assert np.array_equal(tau[j], t1[0]) and np.array_equal(tb[j], tb1[0]) and np.array_equal(dl[j], dl1[0])


@pytest.mark.gpu
def test_digit_products_are_taken(solver_factory):
    """A 64-column step that leaves at least 384 rows updates them by digit products: four launches
    instead of one."""
    s = solver_factory(3, 1, 1)
    energies = W.semicircle_contour(-0.2, 0.7, 2)
    probs = _register(s, (3, 5, 7), energies)
    count = []
    for a, p in enumerate(probs):
        s.solve_jobs(T.make_jobs([(a, i, 0, e) for i, e in enumerate(energies)]), T.PREC_FP64)
        steps = [p.nrmat_ns - k - 64 for k in range(0, p.nrmat_ns - 16, 64)]
        # W, the next diagonal block, its inverse and the update for every step but the last
        count.append((s.last_launch_count, 4 * len(steps) + 3 * sum(m >= 384 for m in steps)))
    assert count[1][0] - count[0][0] == count[1][1] - count[0][1]
    assert count[2][0] - count[0][0] == count[2][1] - count[0][1]


@pytest.mark.gpu
@pytest.mark.parametrize("s", [0, 25, 60])
def test_balance_of_the_inner_indices(solver_factory, s):
    """The first block's rows and columns scaled against each other by 2^s and 2^-s in turn, which leaves
    tau00 as it is.  Digits scaled by row and by column alone would keep 62 - 2 s bits of the small half
    of the operands."""
    rng = np.random.default_rng(s)
    n, b = 1040, 16
    m = np.eye(n) + 0.3 / np.sqrt(n) * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
    first = slice(b, b + 64)  # the rows eliminated first
    m[first, first] = np.eye(64)
    t0 = rng.normal(size=(b, b)) + 1j * rng.normal(size=(b, b))
    rhs = np.zeros((n, b), np.complex128)
    rhs[:b] = t0
    want = np.linalg.solve(m, rhs)[:b]
    e = np.zeros(n, np.int64)
    e[first] = np.where(np.arange(64) % 2 == 0, s, -s)
    f = np.ldexp(1.0, e)
    x = solver_factory(3, 1, 1)
    x.set_refinement(T.PREC_FP64, 0)
    try:
        got = x.solve_tau00_dense(m * f[:, None] / f[None, :], t0, T.PREC_FP64)
    finally:
        x.set_refinement(T.PREC_FP64, 1)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.gpu
def test_panel_pivoting_with_digit_products(solver_factory):
    """Rows in random order at a size whose first steps take the digit products."""
    m, t0, want = _dense(16 + 1101, 16, 7, shuffle=True)
    s = solver_factory(3, 1, 1)
    s.set_pivoting(T.PIVOT_PANEL)
    try:
        got = s.solve_tau00_dense(m, t0, T.PREC_FP64)
    finally:
        s.set_pivoting(T.PIVOT_AUTO)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("b,rest", [(32, 321), (32, 700), (9, 321), (16, 65)])
def test_accelerated_rounds_of_an_ill_conditioned_matrix(solver_factory, b, rest):
    """Condition number 1e5: several accelerated rounds, odd N and 32 columns among them."""
    n = b + rest
    rng = np.random.default_rng(n)
    q = [np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))[0] for _ in range(2)]
    m = (q[0] * np.logspace(0, -5, n)) @ q[1]
    t0 = rng.normal(size=(b, b)) + 1j * rng.normal(size=(b, b))
    rhs = np.zeros((n, b), np.complex128)
    rhs[:b] = t0
    want = np.linalg.solve(m, rhs)[:b]
    got = solver_factory(3, 1, 1).solve_tau00_dense(m, t0, T.PREC_MIXED)
    assert np.abs(got - want).max() <= TOL_MIXED * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("pivoting", [T.PIVOT_BLOCK, T.PIVOT_PANEL])
@pytest.mark.parametrize("min_rest", [1, 512])
def test_paired_steps_of_uneven_waves(solver_factory, min_rest, pivoting):
    """Mixed waves whose smaller jobs end in a partial block at what would be a pair's second step (N = 1392
    beside 2160: n = 21 x 64 + 32): every job refines, and to the FP64 result."""
    s = solver_factory(3, 1, 1)
    energies = W.semicircle_contour(-0.2, 0.7, 4)
    _register(s, (6, 7, 4), energies)
    jobs = T.make_jobs([(a, i, 0, e) for i, e in enumerate(energies) for a in range(3)])
    want = s.solve_jobs(jobs, T.PREC_FP64)
    s.set_pivoting(pivoting)
    s.set_paired_steps(min_rest)
    try:
        got = s.solve_jobs(jobs, T.PREC_MIXED)
        assert s.last_fallback_count == 0
    finally:
        s.set_paired_steps(768)
        s.set_pivoting(T.PIVOT_AUTO)
    assert np.all(np.abs(got - want).max(axis=1) <= TOL_MIXED * np.abs(want).max(axis=1))

"""Workloads of the tau00 solve that the timing harness measures.

Every case is one energy group of an LSMS energy-contour loop: the program keeps one solver handle and
its registered LIZ geometries, uploads the group's single-site t-matrices and solves every (energy,
spin, atom) of the group (``TauSolver.upload_tmat`` + the solve entry).  Inputs are the synthetic
phase-shift t-matrices of ``lsms_b200.workloads`` (phase shifts U(0, 1.2), 5% vacancies with
U(0, 0.05), a random moment per site for non-collinear spin) on bcc (a = 5.42 bohr) and fcc
(a = 6.82 bohr) LIZ geometries, over the semicircular contour from -0.3 to 0.7 Ry.

Fields of a case
  kind      "tau" (tau00_l), "vjp" (adjoint of tau00 and ln det M), "full" (tau over the whole LIZ)
  lattice   "bcc" or "fcc"
  shells    coordination shells of the LIZ; 0: uneven, atom a takes 3 + a % 5 shells
  outer_l   lmax of the outer half of the LIZ sites (3: no step)
  cant      n_spin_cant (2: non-collinear, blocks of 32);  pola: n_spin_pola
  atoms, energies   size of the group;  extra: add the point etop + 0.0025 i to the contour
  mixed     FP32 factors with FP64 refinement instead of plain FP64
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from lsms_b200 import tau as T
from lsms_b200 import workloads as W

_LMAX = 3
_KK = (_LMAX + 1) ** 2
_A = {"bcc": 5.42, "fcc": 6.82}


def _case(name=None, **kw):
    c = {} if name is None else {"name": name}
    c.update(kind="tau", lattice="fcc", shells=7, outer_l=3, cant=1, pola=1, atoms=1, energies=1, extra=False,
             mixed=False)
    c.update(kw)
    return c


def listed():
    return [
        # one site, one energy of the smallest configuration (bcc, 15 sites, N = 240): a call's latency
        _case("site_n240", lattice="bcc", shells=2),
        # both spins of a collinear-polarised contour, LIZ with an lmax step (N = 156)
        _case("spins_n156", lattice="bcc", shells=2, outer_l=1, pola=2, energies=31),
        # one (atom, energy) per call at N = 2160, the reference's calling pattern
        _case("energy_n2160_fp64"),
        _case("energy_n2160_mixed", mixed=True),
        # a whole 31-point contour of one atom at N = 2160, the benchmark's workload
        _case("contour_n2160_fp64", energies=31),
        _case("contour_n2160_mixed", energies=31, mixed=True),
        # local atoms with LIZ sizes 43 ... 135 (N = 688 ... 2160) in one batch
        _case("uneven_fp64", shells=0, atoms=8, energies=8),
        _case("uneven_mixed", shells=0, atoms=8, energies=32, extra=True, mixed=True),
        # non-collinear spin: the largest LIZ (N = 4320) mixed, a small one (N = 1376) in FP64
        _case("noncollinear_n4320_mixed", cant=2, pola=2, energies=16, mixed=True),
        _case("noncollinear_n1376_fp64", shells=3, cant=2, pola=2, energies=8),
        # derivatives with respect to every site's t-matrix (N = 1392)
        _case("adjoint_n1392", kind="vjp", shells=6, energies=16),
        # tau over the whole LIZ for the Kubo current matrix (N = 880)
        _case("full_n880", kind="full", shells=4),
    ]


def draw(rng):
    kind = rng.choice(["tau"] * 8 + ["vjp", "full"])
    c = _case(kind=kind, lattice=rng.choice(["bcc", "fcc"]), outer_l=rng.choice([3, 3, 1, 2]))
    c["cant"], c["pola"] = rng.choice([(1, 1), (1, 1), (1, 2), (2, 2)])
    c["mixed"] = kind == "tau" and rng.random() < 0.5
    if c["mixed"] and c["cant"] == 1 and c["outer_l"] == 2:
        c["outer_l"] = 1  # mixed cases have an even N: blocks of 16 and 4, not 9
    c["shells"] = rng.randint(1, 7) if kind == "tau" else rng.randint(1, 5)
    if kind == "tau" and rng.random() < 0.25:
        c["shells"] = 0
        c["atoms"] = rng.randint(2, 8)
    if kind != "full":
        # at most what a contour at N = 2160 costs in plain FP64, four times that mixed
        most = 8.5e11 * (4 if c["mixed"] else 1)
        one = work(dict(c, energies=1))["flops"]
        top = int(max(1, min(32, most / one)))
        c["energies"] = min(top, max(1, round(math.exp(rng.uniform(0.0, math.log(top + 0.5))))))
        if kind == "vjp":
            c["energies"] = min(c["energies"], 16)
        c["extra"] = c["energies"] > 8 and rng.random() < 0.3
    return c


# --- the inputs -----------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _lattice(lattice, shells):
    return W.lattice_shells(lattice, _A[lattice], shells)


def _geometry(case, a):
    """Positions (3, L) and per-site lmax of local atom a."""
    pos = _lattice(case["lattice"], case["shells"] or 3 + a % 5)
    lmax = np.full(pos.shape[1], _LMAX, np.int32)
    lmax[(pos.shape[1] + 1) // 2:] = case["outer_l"]
    return pos, lmax


def _energies(case):
    n = case["energies"]
    if n == 1:
        return np.array([0.35 + 0.15j])
    return W.semicircle_contour(-0.3, 0.7, n - 1 if case["extra"] else n, extra_point=case["extra"])


def _inputs(case, seed):
    """The group's energies, tmatStore (nstore, energies, blk), spin frames and per-atom LIZ."""
    rng = np.random.default_rng([seed, 17])
    e = _energies(case)
    prel = np.array([W.prel_of(x) for x in e])
    own = case["cant"] == 2 or case["kind"] == "vjp"  # a store column per site, else two species + vacancy
    geo = [_geometry(case, a) for a in range(case["atoms"])]
    nstore = max(p.shape[1] for p, _ in geo) if own else 3
    delta = rng.uniform(0.0, 1.2, size=(nstore, 2, _LMAX + 1))
    if not own:
        delta[2] = rng.uniform(0.0, 0.05, size=(2, _LMAX + 1))
    ev = rng.normal(size=(nstore, 3))
    ev /= np.linalg.norm(ev, axis=1, keepdims=True)
    lof = np.repeat(np.arange(_LMAX + 1), 2 * np.arange(_LMAX + 1) + 1)
    # t of every (column, energy, spin, L)
    td = (-(1.0 / prel)[None, :, None, None] * (np.sin(delta) * np.exp(1j * delta))[:, None])[..., lof]
    blk = (2 * _KK) ** 2
    store = torch.zeros((nstore, len(e), blk), dtype=torch.complex128, pin_memory=torch.cuda.is_available()).numpy()
    frames = [W.spin_trafo(v) for v in ev]
    d = np.arange(_KK)
    if case["cant"] == 2:
        t = store.reshape(nstore, len(e), 2 * _KK, 2 * _KK)  # [column][row] of the b x b block
        for s, (u, ud) in enumerate(frames):
            um, udm = u.reshape(2, 2, order="F"), ud.reshape(2, 2, order="F")
            for i in range(2):
                for j in range(2):
                    t[s][:, j * _KK + d, i * _KK + d] = sum(udm[i, p] * td[s, :, p] * um[p, j] for p in range(2))
    else:
        for s in range(case["pola"]):
            store[:, :, s * _KK * _KK + d * _KK + d] = td[:, :, s]
    atoms = []
    for a, (pos, lmax) in enumerate(geo):
        L = pos.shape[1]
        if own:
            idx = (np.arange(L) + 7 * a) % nstore
        else:
            idx = rng.choice(3, size=L, p=[0.475, 0.475, 0.05])
            idx[0] = rng.integers(0, 2)
        atoms.append((pos, lmax, idx.astype(np.int32)) + frames[idx[0]])
    b = case["cant"] * _KK
    bar = rng.normal(size=(len(e) * case["atoms"], b, b, 2)) @ np.array([1.0, 1j])
    return {"energies": e, "prel": prel, "store": store, "atoms": atoms, "taubar": bar}


_program = {}  # the running program's handle: its solver and the number of LIZ registered on it


def prepare(case, seed):
    s = _inputs(case, seed)
    key = sorted((k, v) for k, v in case.items() if k != "name")
    if _program.get("key") != key:
        _program.clear()
        _program.update(key=key, solver=T.TauSolver(_LMAX, case["cant"], case["pola"]), used=0)
    s["case"], s["solver"] = case, _program["solver"]
    s["ids"] = list(range(_program["used"], _program["used"] + case["atoms"]))
    _program["used"] += case["atoms"]
    for i, (pos, lmax, idx, u, ud) in zip(s["ids"], s["atoms"]):
        s["solver"].set_atom(i, pos, lmax, idx, u, ud)
    return s


def run(state):
    s, case, e = state["solver"], state["case"], state["energies"]
    prec = T.PREC_MIXED if case["mixed"] else T.PREC_FP64
    s.upload_tmat(state["store"])
    if case["kind"] == "full":
        a = state["ids"][0]
        return s.solve_tau_full(a, 0, 0, e[0], s.atom_n[a])
    if case["kind"] == "vjp":
        jobs = T.make_jobs([(a, i, 0, x) for i, x in enumerate(e) for a in state["ids"]])
        num = [a[0].shape[1] for a in state["atoms"]] * len(e)
        return s.solve_vjp(jobs, state["taubar"], num)
    if len(e) == 1 and case["atoms"] == 1 and _nspin(case) == 1:
        return s.calculate_tau_matrix(state["ids"][0], 0, e[0], 0, prec)
    return s.calculate_all_tau_matrices(state["ids"], e, prec=prec)


def _nspin(case):
    return 2 if case["kind"] == "tau" and case["pola"] != case["cant"] else 1


def work(case):
    """Real operations of the block elimination and build (refinement not counted), and the t-matrices,
    LIZ positions and results once."""
    flops = nbytes = 0.0
    b = case["cant"] * _KK
    nspin = _nspin(case)
    for a in range(case["atoms"]):
        pos, lmax = _geometry(case, a)
        L = len(lmax)
        N = case["cant"] * float(((lmax + 1) ** 2).sum())
        n = N - b
        f = 8 * N * N + 8.0 / 3 * n ** 3 + 8 * n * n * b + 8 * n * b * b + 8.0 / 3 * b ** 3 + 8 * b ** 3
        out = b * b
        if case["kind"] == "vjp":  # the inverse from the factors, and the products per site
            f += 16.0 / 3 * N ** 3 + 8 * N * N * 2 * b + 8 * N * b * b
            out += 2 * L * b * b
        elif case["kind"] == "full":
            f = 8 * N * N + 8 * N ** 3 + 8 * N * N * b
            out = N * N
        jobs = case["energies"] * nspin
        flops += jobs * f
        nbytes += jobs * 16.0 * (L * b * b + out) + 24.0 * L
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Two correct FP64 solves differ by about the condition number (up to some 1e6 here) times 1e-16,
    and the adjoint applies the inverse twice.  Against exact(), over 600 runs of these ranges: tau00
    to 3e-11, full tau to 1.4e-10, gradients to 4e-9 (largest element 1.3e-9, 4e-9, 2e-7 of the rms)."""
    return {"rel": 2e-8, "max": 1e-6} if case["kind"] == "vjp" else {"rel": 6e-10, "max": 2e-8}


# --- the same results in 64 bits by dense linear algebra ---------------------------------------------

def _pbar(x, top):
    """Normalised associated Legendre functions P_lm(x), Condon-Shortley phase, m >= 0."""
    y = torch.sqrt(1.0 - x * x)
    p = {(0, 0): torch.full_like(x, math.sqrt(0.25 / math.pi))}
    for m in range(1, top + 1):
        p[m, m] = -math.sqrt((2 * m + 1) / (2 * m)) * y * p[m - 1, m - 1]
    for m in range(top + 1):
        for l in range(m + 1, top + 1):
            a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
            b = math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1)) if l > m + 1 else 0.0
            p[l, m] = a * (x * p[l - 1, m] - (b * p[l - 2, m] if l > m + 1 else 0.0))
    return p


def _signed(p, l, m):
    return p[l, m] if m >= 0 else (-1) ** m * p[l, -m]


@functools.lru_cache(maxsize=None)
def _coupling():
    """(49, 256): G(lm2, lm1) = sum over (l3, m3) of this times D(l3, m3)."""
    x, w = (torch.from_numpy(v) for v in np.polynomial.legendre.leggauss(20))
    p = _pbar(x, 2 * _LMAX)
    lm = [(l, m) for l in range(_LMAX + 1) for m in range(-l, l + 1)]
    c = torch.zeros(((2 * _LMAX + 1) ** 2, _KK, _KK), dtype=torch.complex128)
    for i2, (l2, m2) in enumerate(lm):
        for i1, (l1, m1) in enumerate(lm):
            m3 = m2 - m1
            for l3 in range(max(abs(m3), abs(l1 - l2)), l1 + l2 + 1):
                if (l1 + l2 + l3) % 2 == 0:
                    g = 2 * math.pi * float((w * _signed(p, l1, m1) * _signed(p, l2, m2) * _signed(p, l3, m3)).sum())
                    c[l3 * (l3 + 1) + m3, i2, i1] = 4 * math.pi * 1j ** (l2 - l1) * g
    return c.reshape(-1, _KK * _KK)


def _structure(pos, prel, dev):
    """G_ij of all site pairs, (L, 16, L, 16), zero for i = j."""
    r = torch.tensor(pos.T.copy(), device=dev)
    L = r.shape[0]
    d = (r[:, None] - r[None, :]).reshape(-1, 3)
    same = torch.eye(L, dtype=torch.bool, device=dev).reshape(-1)
    d[same] = 1.0
    R = d.square().sum(1).sqrt()
    z = prel * R
    h = [torch.full_like(z, -1j), -1.0 - 1j / z]
    for l in range(1, 2 * _LMAX):
        h.append((2 * l + 1) * h[l] / z - h[l - 1])
    p = _pbar(d[:, 2] / R, 2 * _LMAX)
    rho = d[:, :2].square().sum(1).sqrt()
    ok = rho > 1e-6
    ph = torch.where(ok, torch.complex(d[:, 0], d[:, 1]) / torch.where(ok, rho, torch.ones_like(rho)), torch.zeros_like(z))
    phm = [torch.ones_like(ph)]
    for m in range(2 * _LMAX):
        phm.append(phm[m] * ph)
    D = torch.zeros((d.shape[0], (2 * _LMAX + 1) ** 2), dtype=torch.complex128, device=dev)
    for l in range(2 * _LMAX + 1):
        hl = -h[l] * torch.exp(1j * z) / R * 1j ** (l + 1)
        for m in range(l + 1):
            f = p[l, m] * phm[m]
            D[:, l * (l + 1) + m] = hl * f.conj()
            D[:, l * (l + 1) - m] = hl * (-1) ** m * f
    g = D @ _coupling().to(dev)
    g[same] = 0.0
    return g.reshape(L, L, _KK, _KK).permute(0, 2, 1, 3)


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    dev = "cuda"
    s = _inputs(case, seed)
    cant, b = case["cant"], case["cant"] * _KK
    nspin = _nspin(case)
    taus, bars, dets, njob = [], [], [], 0
    for ie in range(len(s["energies"])):
        for isp in range(nspin):
            for pos, lmax, idx, u, ud in s["atoms"]:
                L = pos.shape[1]
                off = isp * _KK * _KK
                t = torch.tensor(s["store"][idx, ie, off:off + b * b], device=dev).reshape(L, b, b).transpose(1, 2)
                G = _structure(pos, complex(s["prel"][ie]), dev)
                big = torch.zeros((L, cant, _KK, L, cant, _KK), dtype=torch.complex128, device=dev)
                for q in range(cant):
                    big[:, q, :, :, q, :] = G
                G = big.reshape(L, b, L * b)
                keep = torch.cat([torch.arange(_KK).repeat(cant) < (int(l) + 1) ** 2 for l in lmax]).to(dev)
                M = (-torch.bmm(t, G)).reshape(L * b, L * b)
                M.diagonal().add_(1.0)
                M = M[keep][:, keep]
                t0 = t[0]
                if case["kind"] == "full":
                    tt = torch.block_diag(*t)[keep][:, keep]
                    return (torch.linalg.inv(M) @ tt).cpu().numpy()
                rhs = torch.zeros((M.shape[0], b), dtype=torch.complex128, device=dev)
                rhs[:b] = t0
                if case["kind"] == "tau":
                    d = torch.linalg.solve(M, rhs)[:b] - t0
                    if cant == 2:
                        U = torch.tensor(u.reshape(2, 2, order="F"), device=dev)
                        V = torch.tensor(ud.reshape(2, 2, order="F"), device=dev)
                        q = torch.einsum("ap,pxqy,qc->caxy", U, d.reshape(2, _KK, 2, _KK), V)
                        taus.append(q.transpose(2, 3).reshape(-1))
                    else:
                        taus.append(d.T.reshape(-1))
                    continue
                V = torch.linalg.inv(M)
                X = V @ rhs
                G = G.reshape(L * b, L * b)[keep][:, keep]
                bar = torch.tensor(s["taubar"][njob], device=dev)
                njob += 1
                lam, Z, H = V[:b].T @ bar, G @ X, G @ V
                taus.append(X[:b])
                at = torch.cumsum(torch.tensor([0] + [cant * (int(l) + 1) ** 2 for l in lmax]), 0).tolist()
                gb = torch.zeros((L, b, b), dtype=torch.complex128, device=dev)
                gd = torch.zeros_like(gb)
                kept = keep.reshape(L, b)
                for j in range(L):
                    r = slice(at[j], at[j + 1])
                    w = torch.nonzero(kept[j]).reshape(-1)
                    tb = lam[r] @ Z[r].T + (lam[r] if j == 0 else 0.0)
                    gb[j, w[:, None], w[None, :]] = tb
                    gd[j, w[:, None], w[None, :]] = -H[r, r].T
                bars.append(gb.cpu().numpy())
                dets.append(gd.cpu().numpy())
    if case["kind"] == "vjp":
        return torch.stack(taus).cpu().numpy(), bars, dets
    taus = torch.stack(taus).reshape(len(s["energies"]), nspin, len(s["atoms"]), -1)
    if len(s["energies"]) == 1 and case["atoms"] == 1 and nspin == 1:
        taus = taus.reshape(-1)
    return taus.cpu().numpy()

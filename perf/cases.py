"""What the speed of this library is measured on: the calls a user's program makes through the handler
(correlation energy, chi0(q, omega), exchange, G0W0), from the smallest cells to the largest a pass of
two seconds takes.

A case is a system and the call made on it.  Systems are seeded synthetic inputs of the benchmark's
distributions (librpa_gb300/synthetic.py): KS energies uniform in [-0.8, -0.2] Ha and [0.1, 2.0] Ha,
random unitary eigenvectors, RI coefficients Gaussian * exp(-d / decay), V(q) = A A^H + 0.1, and the
minimax window that goes with the number of points.  `species` lists NAO/ABF counts per atom, dealt
round-robin, so that a case's shapes do not depend on the seed.

The FP64 calls return double precision.  The default calls form their products from BF16 pieces
accumulated in FP32 (E_c is good to about 1e-6 relative, and its last digits move with the launch
shape the library's tuner picks), so their results are kept in single precision.
"""
import ctypes
import math
import os
from types import SimpleNamespace

import numpy as np
import torch

import librpa_gb300 as L

ANGSTROM = 1.8897259886
EMIN, RANGE = 0.25, {16: 100.0, 24: 3000.0, 32: 10000.0}
PRECISION = {"split": L.CHI0_BF16X3, "fp32": L.CHI0_FP32, "fp64": L.CHI0_FP64}
EC_PATH = {"chol": L.EC_CHOL, "chol_fp64": L.EC_CHOL_FP64, "lu": L.EC_LU_FP64}
SIGMA = {"fp64": L.SIGMA_FP64, "split": L.SIGMA_BF16X3}
MIXED = "5/20,13/60,26/110"


def _case(name, call, atoms, species, k=(1, 1, 1), nfreq=16, **kw):
    c = dict(call=call, atoms=atoms, species=species, k1=k[0], k2=k[1], k3=k[2], nfreq=nfreq, spins=1, ibz=False,
             half_bands=False, decay=2.0, precision="split", ec="chol", sigma="fp64", cells=1)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a molecule in a box: the smallest call, all latency and launches
        _case("ec_molecule", "ec", 3, MIXED, nfreq=24),
        # a scan over small molecules of 2 to 8 atoms, one batched call
        _case("ec_batch", "batch", 8, MIXED, nfreq=24, cells=12),
        # the 2-atom fcc cell on its 2x2x2 k-mesh
        _case("ec_fcc2_k222", "ec", 2, "13/40", (2, 2, 2)),
        # the 16-atom supercell on 3x3x3 k-points: the benchmark's headline call
        _case("ec_fcc16_k333", "ec", 16, "13/40", (3, 3, 3), half_bands=True),
        # a large cell of mixed species at Gamma (48 of the 64 atoms of the benchmark's: two seconds a pass)
        _case("ec_mixed48", "ec", 48, MIXED, nfreq=24),
        # 128 atoms at Gamma, short-ranged RI coefficients
        _case("ec_gamma128", "ec", 128, "13/40", decay=1.5),
        # atoms with more orbitals than the tensor-core tiles hold
        _case("ec_large_atoms", "ec", 6, "36/140,13/60"),
        # the all-FP64 reference form, for parity runs
        _case("ec_fp64_fcc2_k222", "ec", 2, "13/40", (2, 2, 2), precision="fp64", ec="lu"),
        # chi0(q, omega) alone (a tau- or q-sharded program), spin-polarised, ragged sizes, odd mesh, IBZ q points
        _case("chi0_ragged_k331", "chi0", 3, "9/31,14/47,5/18", (3, 3, 1), spins=2, ibz=True),
        # exchange of a k-grid, all states
        _case("exx_fcc2_k222", "exx", 2, "13/40", (2, 2, 2)),
        # G0W0 self-energy of a molecule in FP64 throughout
        _case("g0w0_molecule", "g0w0", 3, "13/40,5/20", precision="fp64", ec="lu"),
        # G0W0 self-energy on a k-grid with the library's default precisions
        _case("g0w0_k221", "g0w0", 2, "5/20,9/31", (2, 2, 1)),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def between(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    call = rng.choice(["ec", "ec", "ec", "ec_k", "ec_k", "ec_fp64", "batch", "chi0", "exx", "g0w0"])
    nfreq = rng.choice([16, 24])
    few = ["13/40", "5/20", "5/20,13/60", MIXED, "9/31,14/47,5/18", "%d/%d" % (rng.randint(4, 16), rng.randint(15, 60))]
    if call == "ec":
        species = rng.choice(few[:-1])
        return _case(None, "ec", between(2, 96 if species == "13/40" else 48), species, nfreq=nfreq, decay=rng.choice([1.5, 2.0]))
    if call == "ec_k":
        k = rng.choice([(2, 1, 1), (2, 2, 2), (3, 1, 1), (3, 3, 1), (3, 2, 1)])
        return _case(None, "ec", between(2, 64 // (k[0] * k[1] * k[2]) + 2), rng.choice(few), k, nfreq,
                     ibz=rng.random() < 0.5, spins=rng.choice([1, 1, 2]), half_bands=rng.random() < 0.5)
    if call == "ec_fp64":
        return _case(None, "ec", rng.randint(2, 6), "%d/%d" % (rng.randint(5, 13), rng.randint(18, 40)), nfreq=16,
                     precision="fp64", ec=rng.choice(["lu", "chol_fp64"]))
    if call == "batch":
        return _case(None, "batch", rng.randint(3, 8), rng.choice([MIXED, "5/20,13/60"]), nfreq=nfreq, cells=between(2, 16))
    if call == "chi0":
        k = rng.choice([(1, 1, 1), (2, 2, 1), (3, 3, 1), (2, 2, 2)])
        return _case(None, "chi0", rng.randint(2, 5), rng.choice(few), k, nfreq, spins=rng.choice([1, 2]),
                     ibz=rng.random() < 0.5, precision=rng.choice(["split", "split", "fp32"]))
    if call == "exx":
        k = rng.choice([(1, 1, 1), (2, 1, 1), (2, 2, 1), (2, 2, 2), (3, 2, 1)])
        return _case(None, "exx", rng.randint(2, 3), rng.choice(["13/40", "5/20", "9/31,5/18"]), k)
    k = rng.choice([(1, 1, 1), (1, 1, 1), (2, 1, 1), (2, 2, 1)])
    return _case(None, "g0w0", 2, rng.choice(["5/20,9/31", "5/20", "7/25"]), k, precision=rng.choice(["split", "fp64"]),
                 sigma=rng.choice(["fp64", "fp64", "split"]))


# ------------------------------------------------------------------ inputs
def _sizes(case, atoms):
    sp = [tuple(int(x) for x in s.split("/")) for s in case["species"].split(",")]
    return [sp[i % len(sp)][0] for i in range(atoms)], [sp[i % len(sp)][1] for i in range(atoms)]


def _atoms(case):
    """Atoms of each cell of the case: one cell, or a batch of cells of 2 atoms up to `atoms`."""
    if case["call"] != "batch":
        return [case["atoms"]]
    return [2 + (5 * i) % (case["atoms"] - 1) for i in range(case["cells"])]


def _geometry(atoms, gamma):
    """Lattice (rows, Bohr) and positions: the fcc diamond cell and its supercells, else a cubic packing."""
    s = round((atoms / 2) ** (1 / 3))
    if not gamma and 2 * s ** 3 == atoms:
        a = 3.57 * ANGSTROM
        lat = 0.5 * a * np.array([[0.0, 1, 1], [1, 0, 1], [1, 1, 0]])
        base = np.array([[0.0, 0, 0], [0.25 * a] * 3])
        pos = np.concatenate([base + i * lat[0] + j * lat[1] + k * lat[2] for i in range(s) for j in range(s) for k in range(s)])
        return s * lat, pos
    side = math.ceil(atoms ** (1 / 3) - 1e-9)
    pos = np.array([(i, j, k) for i in range(side) for j in range(side) for k in range(side)][:atoms], float)
    step = 2.5 * ANGSTROM
    return np.eye(3) * (side * step + (20.0 * ANGSTROM if gamma else 0.0)), pos * step


def _mesh(n):
    """Fractional k-points and, for each, the index of -k."""
    fr = [(i, j, l) for i in range(n[0]) for j in range(n[1]) for l in range(n[2])]
    at = {f: i for i, f in enumerate(fr)}
    partner = np.array([at[tuple((-x) % p for x, p in zip(f, n))] for f in fr])
    return np.array(fr, float) / np.array(n, float), partner


def _cells(n):
    return [(x, y, z) for x in range(-(n[0] // 2), (n[0] - 1) // 2 + 1) for y in range(-(n[1] // 2), (n[1] - 1) // 2 + 1)
            for z in range(-(n[2] // 2), (n[2] - 1) // 2 + 1)]


def _system(case, seed, atoms):
    """The record librpa_gb300.load_system takes; random numbers are drawn on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    nao, nabf = _sizes(case, atoms)
    n = (case["k1"], case["k2"], case["k3"])
    fr, partner = _mesh(n)
    nk, ns, tao, N = len(fr), case["spins"], sum(nao), sum(nabf)
    lat, pos = _geometry(atoms, nk == 1)
    recip = 2.0 * math.pi * np.linalg.inv(lat).T
    nb = tao // 2 if case["half_bands"] else tao
    nocc = max(1, tao // 13 if nk > 1 else tao // 4)

    def uniform(lo, hi, shape):
        return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)

    def normal(shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)

    ekb = torch.cat([uniform(-0.8, -0.2, (ns, nk, nocc)).sort().values, uniform(0.1, 2.0, (ns, nk, nb - nocc)).sort().values], 2)
    ekb = ekb.cpu().numpy()
    wfc = np.zeros((ns, nk, nb, tao), complex)
    Vk = {}
    for k in range(nk):
        p = int(partner[k])
        if p < k:  # time reversal
            ekb[:, k], wfc[:, k], Vk[k] = ekb[:, p], wfc[:, p].conj(), Vk[p].conj()
            continue
        z = normal((ns, tao, nb)) + (0 if p == k else 1j * normal((ns, tao, nb)))
        wfc[:, k] = np.swapaxes(np.linalg.qr(z.cpu().numpy())[0], 1, 2)
        a = normal((N, N)) if p == k else torch.complex(normal((N, N)), normal((N, N)))
        Vk[k] = (a @ a.mH / (N if p == k else N / 2) + 0.1 * torch.eye(N, device="cuda", dtype=torch.float64)).cpu().numpy()
    wg = np.zeros((ns, nk, nb))
    wg[:, :, :nocc] = 2.0 / ns
    cells = _cells(n)
    amp = {}
    for I in range(atoms):
        for J in range(atoms):
            for R in cells:
                d = np.linalg.norm(pos[J] + np.asarray(R, float) @ lat - pos[I])
                amp[I, J, R] = 0.02 * math.exp(-d / (case["decay"] * ANGSTROM))
    count = [nao[I] * nao[J] * nabf[I] for I, J, _ in amp]
    scale = torch.repeat_interleave(torch.tensor(list(amp.values()), device="cuda", dtype=torch.float64),
                                    torch.tensor(count, device="cuda"))
    flat = (normal((sum(count),)) * scale).cpu().numpy()
    del scale
    Cs, o = {}, 0
    for (I, J, R), c in zip(amp, count):
        Cs[I, J, R] = flat[o:o + c].reshape(nao[I] * nao[J], nabf[I])
        o += c
    off = np.concatenate([[0], np.cumsum(nabf)]).astype(int)
    ibz = np.minimum(np.arange(nk), partner) if case["ibz"] else np.arange(nk)
    Vq = {(k, I, J): Vk[k][off[I]:off[I + 1], off[J]:off[J + 1]] for k in sorted(set(ibz.tolist()))
          for I in range(atoms) for J in range(I, atoms)}
    return SimpleNamespace(n_spins=ns, n_kpts=nk, n_bands=nb, n_ao=tao, period=n, latvec=lat, kvecs=fr @ recip, fr=fr,
                           ibz_map=ibz, positions=pos, types=np.arange(atoms) % len(case["species"].split(",")), nao=nao,
                           nabf=nabf, wg=wg, ekb=ekb, efermi=-0.05, wfc=wfc, Cs=Cs, Vq=Vq, Vk=Vk, cells=cells, nocc=nocc,
                           v_cut=Vq if case["call"] in ("exx", "g0w0") else {})


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    """The handlers with their inputs set, as a program has them before the call."""
    hs, nq = [], []
    for i, atoms in enumerate(_atoms(case)):
        s = _system(case, seed * 1000 + i, atoms)
        h = L.Handler()
        L.load_system(h, s)
        h.set_gb300_options(L.gb300_options(
            chi0_precision=PRECISION[case["precision"]], ec_path=EC_PATH[case["ec"]], sigma_precision=SIGMA[case["sigma"]],
            stage=L.STAGE_CHI0 if case["call"] == "chi0" else L.STAGE_FULL))
        hs.append(h)
        nq.append(len(set(s.ibz_map.tolist())))
    nf = case["nfreq"]
    o = L.Options(nfreq=nf, tfgrids_type=L.Minimax, parallel_routing=L.LIBRI, minimax_emin=EMIN, minimax_emax=EMIN * RANGE[nf])
    return SimpleNamespace(call=case["call"], hs=hs, h=hs[0], nq=nq[0], opts=o, spins=case["spins"], nk=s.n_kpts, nb=s.n_bands,
                           nfreq=nf, single=case["precision"] != "fp64")


def run(st):
    h, o = st.h, st.opts
    if st.call == "batch":
        return L.rpa_correlation_energy_batch(st.hs, o).astype(np.float32)
    if st.call == "ec":
        ec, per_q = h.get_rpa_correlation_energy(o, st.nq)
        return {"ec": np.float32(ec), "per_q": per_q.astype(np.complex64)} if st.single else {"ec": np.float64(ec), "per_q": per_q}
    if st.call == "chi0":
        h.get_rpa_correlation_energy(o, st.nq)
        t = h.chi0_qw_tensor("cuda")
        return t.float() if st.single else t
    if st.call == "exx":
        h.lib.librpa_build_exx(h.h, ctypes.byref(o))
        h._check()
        return h.get_exx_pot_kgrid(o, st.spins, list(range(st.nk)), 0, st.nb)
    h.lib.librpa_build_g0w0_sigma(h.h, ctypes.byref(o))
    h._check()
    sig = np.stack([[h.g0w0_sigc_iw(s, 0, st.nb, st.nfreq, k) for k in range(st.nk)] for s in range(st.spins)])
    return sig.astype(np.complex64) if st.single else sig


# ------------------------------------------------------------------ the work a pass cannot do without
def _work_one(case, atoms):
    nao, nabf = _sizes(case, atoms)
    n = case["k1"] * case["k2"] * case["k3"]
    tao, N, ns, nw = sum(nao), sum(nabf), case["spins"], case["nfreq"]
    nb = tao // 2 if case["half_bands"] else tao
    cx = 1 if n == 1 else 4  # real multiply-adds of one complex one
    nq = n if not case["ibz"] else len(set(np.minimum(np.arange(n), _mesh((case["k1"], case["k2"], case["k3"]))[1]).tolist()))
    sup, rows = n * tao, sum(a * b for a, b in zip(nao, nabf))
    chi = 4.0 * rows * sup * sup
    for I in range(atoms):
        for J in range(I, atoms):
            aI, aJ, bI, bJ = nao[I], nao[J], nabf[I], nabf[J]
            chi += n * 4.0 * (bI * aI * aJ * sup + bI * bJ * aJ * sup / 2 + bI * bJ * aI * aJ)
    chi *= nw * ns
    pairs = sum(nabf[I] * nabf[J] for I in range(atoms) for J in range(I, atoms))
    read = 8.0 * rows * sup + 16.0 * ns * n * nb * tao + 16.0 * nq * pairs
    if case["call"] in ("ec", "batch"):
        return read + 16.0 * nq, chi + nq * nw * cx * (4.0 * N ** 3 + N ** 3 / 3.0)
    if case["call"] == "chi0":
        return read + 16.0 * nw * nq * pairs, chi
    # H of one cell's rows: U D, W times that, and the contraction with U over the supercell
    hs = 2.0 * n * N * sup * sup * tao + 2.0 * (n * N) ** 2 * tao * sup + 2.0 * n * N * sup * sup * tao
    if case["call"] == "exx":
        return read + 8.0 * ns * n * nb, ns * hs
    wc = nq * nw * cx * (8.0 * N ** 3 + 8.0 * N ** 3 / 3.0)
    return read + 16.0 * nq * pairs + 16.0 * ns * n * nb * nw, chi + wc + 2 * ns * nw * hs


def work(case):
    w = [_work_one(case, a) for a in _atoms(case)]
    return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch
def _minimax(n):
    """GreenX's minimax nodes and least-squares transform weights (the library's tables, numpy's SVD)."""
    path = os.path.join(os.path.dirname(L.__file__), "data", "greenx_minimax_tables.txt")
    emin, emax = EMIN, EMIN * RANGE[n]
    er, cols, kind = {}, {}, None
    for line in open(path):
        t = line.split()
        if not t or t[0].startswith("#"):
            continue
        if t[0] == "table":
            kind = t[1] if int(t[2]) == n else None
        elif kind and t[0] == "erange":
            er[kind] = [float(x) for x in t[1:]]
        elif kind and t[0] == "col":
            cols[kind, int(t[1])] = np.array([float(x) for x in t[2:]])

    def nodes(kind):
        up = [j for j, v in enumerate(er[kind], 1) if emax / emin < v]
        i, ratio = (min(up, key=lambda j: er[kind][j - 1]) if up else len(er[kind]) + 1), 1.0
        if i == 1 and n > 20:
            ratio = er[kind][0] / (emax / emin)
            ratio = ratio / 1.5 if ratio > 1.5 else ratio
        c = cols[kind, i]
        return (c / ratio if kind == "omega" else c * ratio)

    om, ta = nodes("omega") * emin, nodes("tau") / (2 * emin)
    om, wom, ta = om[:n], om[n:], ta[:n]
    m = max((int(math.log10(emax / emin)) + 1) * 200, n)
    x = emin * (emax / emin) ** (np.arange(m) / (m - 1.0))

    def fit(A, y):
        U, S, VT = np.linalg.svd(A, full_matrices=False)
        return VT.T @ ((U.T @ y) / S)

    E = np.exp(-np.outer(x, ta))
    t2f = np.array([np.cos(w * ta) * fit(np.cos(w * ta) * E, 2 * x / (x * x + w * w)) for w in om])
    s2f = np.array([np.sin(w * ta) * fit(np.sin(w * ta) * E, 2 * w / (x * x + w * w)) for w in om])
    F = 2 * x[:, None] / (x[:, None] ** 2 + om[None] ** 2)
    f2t = np.array([np.cos(t * om) * fit(np.cos(t * om) * F, np.exp(-x * t)) for t in ta])
    return om, wom, ta, t2f, f2t, s2f


class _Exact:
    """The supercell of the k-grid in dense form: U[a, p, r] = C_a[p, r] + C_a[r, p] for the ABFs a of the home cell."""

    def __init__(self, s):
        self.s, self.dev = s, torch.device("cuda")
        self.nc, self.N, self.nao = len(s.cells), sum(s.nabf), s.n_ao
        at = {c: i for i, c in enumerate(s.cells)}
        fold = lambda v: tuple((x + p // 2) % p - p // 2 for x, p in zip(v, s.period))  # noqa: E731
        self.c0 = at[(0, 0, 0)]
        self.sub = np.array([[at[fold(np.subtract(a, b).tolist())] for b in s.cells] for a in s.cells])
        self.ph = self.t(np.exp(2j * math.pi * s.fr @ np.array(s.cells, float).T))  # [k][cell]
        ao, ab = np.concatenate([[0], np.cumsum(s.nao)]), np.concatenate([[0], np.cumsum(s.nabf)])
        U = np.zeros((self.N, self.nc * self.nao, self.nc * self.nao))
        for (I, J, R), m in s.Cs.items():
            b = m.reshape(s.nao[I], s.nao[J], s.nabf[I]).transpose(2, 0, 1)
            p, r = self.c0 * self.nao + ao[I], at[R] * self.nao + ao[J]
            U[ab[I]:ab[I + 1], p:p + s.nao[I], r:r + s.nao[J]] += b
            U[ab[I]:ab[I + 1], r:r + s.nao[J], p:p + s.nao[I]] += b.transpose(0, 2, 1)
        self.U, self.ab = self.t(U), ab

    def t(self, a):
        return torch.as_tensor(np.asarray(a), device=self.dev)

    def shifted(self, c):
        """U of the ABFs of cell c."""
        nc, n = self.nc, self.nao
        at = torch.as_tensor(self.sub[:, c], device=self.dev)  # cell d of the supercell, seen from c
        return self.U.view(-1, nc, n, nc, n)[:, at][:, :, :, at].reshape(self.N, nc * n, nc * n)

    def of_r(self, A):
        """Re sum_k e^{-2 pi i k.R} A(k): [cell][.][.]"""
        return torch.einsum("kc,kij->cij", self.ph.conj(), A).real

    def super(self, X):
        """X_s[(c, a)][(d, b)] = X(R_d - R_c)[a][b]"""
        nc, n = X.shape[0], X.shape[1]
        return X[torch.as_tensor(self.sub.T.copy(), device=self.dev)].permute(0, 2, 1, 3).reshape(nc * n, nc * n)

    def density(self, spin, weight):
        w = self.t(self.s.wfc[spin])
        return torch.einsum("kni,kn,knj->kij", w, self.t(weight).to(w.dtype), w.conj())

    def green(self, spin, tau):
        s = self.s
        f, e = s.wg[spin] / s.n_kpts * 0.5 * s.n_spins, s.ekb[spin] - s.efermi
        up = np.exp(np.minimum(0, -tau * e)) * np.maximum(0, 1 / s.n_kpts - f)
        return self.super(self.of_r(self.density(spin, up))), -self.super(self.of_r(self.density(spin, np.exp(np.minimum(0, tau * e)) * f)))

    def chi0(self, grid):
        """chi0(q, omega) [omega][q][N][N] on the IBZ q points."""
        s, (_, _, ta, t2f, _, _) = self.s, grid
        self.q = sorted(set(s.ibz_map.tolist()))
        ph, nn = self.ph[self.q], (self.nc * self.nao) ** 2
        out = torch.zeros(len(ta), len(self.q), self.N, self.N, dtype=torch.complex128, device=self.dev)
        for i, tau in enumerate(ta):
            for spin in range(s.n_spins):
                gp, gm = self.green(spin, tau)
                T = (gp.T @ (self.U @ gm)).reshape(self.N, nn)
                R = torch.stack([T @ self.shifted(c).reshape(self.N, nn).T for c in range(self.nc)])
                X = torch.einsum("qc,cab->qab", ph, R.to(ph.dtype)) * (2.0 / s.n_spins)
                out += self.t(t2f[:, i])[:, None, None, None] * X
        return out

    def closed_form(self, W, D):
        """H_pq = sum U[a,p,r] W[a,b] U[b,q,s] D[r,s] for the rows p of the home cell: [nao][supercell]."""
        home = slice(self.c0 * self.nao, (self.c0 + 1) * self.nao)
        Us = torch.cat([self.shifted(c) for c in range(self.nc)])
        Y = torch.einsum("ab,aps->bps", W, Us[:, home] @ D)
        return torch.einsum("bps,bqs->pq", Y, Us)

    def to_k(self, H):
        """H(k) = sum_c e^{2 pi i k.R_c} H(R_c) on the KS states: [k][state]"""
        H = H.reshape(self.nao, self.nc, self.nao).permute(1, 0, 2)
        return torch.einsum("kc,cij->kij", self.ph, H.to(self.ph.dtype))


def _exact_ec(s, grid):
    x = _Exact(s)
    chi, (_, wom, *_) = x.chi0(grid), grid
    per_q = []
    eye = torch.eye(x.N, device=x.dev, dtype=torch.complex128)
    for i, q in enumerate(x.q):
        A = chi[:, i]
        A = torch.stack([torch.triu(a) + torch.triu(a, 1).mH for a in A])
        P = x.t(s.Vk[q]).to(A.dtype) @ A
        sign, log = torch.linalg.slogdet(eye - P)
        e = torch.log(sign) + log + P.diagonal(dim1=1, dim2=2).sum(1)
        per_q.append(((e * x.t(wom)).sum() * float((s.ibz_map == q).sum()) / s.n_kpts / (2 * math.pi)).item())
    return sum(per_q).real, np.array(per_q)


def _exact_flops(case):
    tot = 0.0
    for atoms in _atoms(case):
        nao, nabf = _sizes(case, atoms)
        n = case["k1"] * case["k2"] * case["k3"]
        sup, N = n * sum(nao), sum(nabf)
        tot += case["spins"] * case["nfreq"] * (4.0 * N * sup ** 3 + 2.0 * n * N * N * sup * sup)
        if case["call"] in ("exx", "g0w0"):
            tot += case["spins"] * case["nfreq"] * 8.0 * n * N * sum(nao) * sup * (sup + n * N)
    return tot


def exact(case, seed):
    if _exact_flops(case) > 8e12:
        return None
    grid = _minimax(case["nfreq"])
    om, wom, ta, t2f, f2t, s2f = grid
    sys = [_system(case, seed * 1000 + i, a) for i, a in enumerate(_atoms(case))]
    if case["call"] == "batch":
        return np.array([_exact_ec(s, grid)[0] for s in sys])
    s = sys[0]
    if case["call"] == "ec":
        ec, per_q = _exact_ec(s, grid)
        return {"ec": np.float64(ec), "per_q": per_q}
    x = _Exact(s)
    if case["call"] == "chi0":
        c, ab, n = x.chi0(grid), x.ab, len(s.nao)
        c = torch.cat([c[:, :, ab[I]:ab[I + 1], ab[J]:ab[J + 1]].flatten(2) for I in range(n) for J in range(I, n)], 2)
        return torch.view_as_real(c.contiguous()).reshape(-1)
    V = x.t(np.stack([s.Vk[k].astype(complex) for k in range(s.n_kpts)]))
    if case["call"] == "exx":
        W, out = x.super(x.of_r(V) / s.n_kpts), []
        for spin in range(s.n_spins):
            D = x.super(x.of_r(x.density(spin, s.wg[spin] / s.n_kpts * 0.5 * s.n_spins)))
            H, w = x.to_k(x.closed_form(W, D)), x.t(s.wfc[spin])
            out.append(-torch.einsum("kni,kij,knj->kn", w.conj(), H, w).real)
        return torch.stack(out).cpu().numpy()
    chi, Wt = x.chi0(grid), 0
    e, Z = torch.linalg.eigh(V)
    S = (Z * e.clamp(min=0).sqrt()[:, None].to(Z.dtype)) @ Z.mH
    eye = torch.eye(x.N, device=x.dev, dtype=torch.complex128)
    for w in range(len(om)):
        A = chi[w]
        A = torch.stack([torch.triu(a) + torch.triu(a, 1).mH for a in A])
        Wc = S @ torch.linalg.inv(eye - S @ A @ S) @ S - S @ S
        Wt = Wt + x.t(f2t[:, w])[:, None, None, None] * x.of_r(Wc)[None] / s.n_kpts
    out = []
    for spin in range(s.n_spins):
        sig, w = 0, x.t(s.wfc[spin])
        for i, tau in enumerate(ta):
            gp, gm = x.green(spin, tau)
            W = x.super(Wt[i])
            hp, hm = (x.to_k(x.closed_form(W, g)) for g in (gp, gm))
            c, sn = (x.t(v[:, i]).to(hp.dtype)[:, None, None, None] for v in (t2f, s2f))
            sig = sig + c * 0.5 * (hp + hm) + 1j * sn * 0.5 * (hp - hm)
        out.append(torch.einsum("kni,wkij,knj->knw", w.conj(), sig, w))
    return torch.stack(out).cpu().numpy()

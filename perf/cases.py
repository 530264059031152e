"""Workloads of the operator library as a program that uses it runs them.

A host that diagonalises H with this library does four things: it uploads the
orbitals of an SCF iteration (set_state), applies the one-, two- and
three-body operators to blocks of trial orbitals (apply, apply_h1), takes the
Davidson subspace step on the device, and, for an optimisation of the Jastrow
factor, asks for the energy gradient.  The cases below run these through
tc_b200.context over the sizes such programs meet: diamond Si with two atoms
(16^3 to 36^3 grids, 1 to 27 k-points), the eight-atom cube on 48^3, the
electron gas, HF / TC / BITC, one and two spin channels, time-reversal
reduced k-sets, double and mixed precision, cubic and uneven grids.

listed() names them, draw() makes more of the same ranges, prepare() builds a
program's state from a seed, run() is one pass, exact() the same numbers from
plain torch in complex128, work() what a pass cannot do without.
"""
import itertools
import math

import numpy as np
import torch

from tc_b200 import abi
from tc_b200.context import Context, davidson_expand, gram_schmidt, subspace_ritz, sum_of_vaux
from tc_b200.system import Pseudo, TCSystem

FOURPI = 4.0 * math.pi
SI_A = 10.26                                     # bohr, lattice constant of silicon
H2_BITS = {"HF": abi.TERM_HF2X | abi.TERM_HF2H, "TC": abi.TERM_TC2X | abi.TERM_TC2H,
           "BITC": abi.TERM_TC2X | abi.TERM_TC2H}
H3_BITS = {"HF": 0, "TC": abi.TERMS_TC & ~abi.TERM_TC2X, "BITC": abi.TERMS_TC & ~abi.TERM_TC2X}


def _case(name, kind, method, cell, mesh, ecut, grid, nocc, nbands, precision, nspin=1, tr=False, channels="equal"):
    return dict(name=name, kind=kind, method=method, cell=cell, mesh=mesh, ecut=ecut, grid=grid, nocc=nocc,
                nbands=nbands, precision=precision, nspin=nspin, tr=tr, channels=channels)


def listed():
    return [
        # one H psi of a Davidson block of a small HF run (3x3x3 mesh, time reversal): host buffers, one- and
        # two-body terms; many short launches
        _case("hf_si2_16_hpsi_fp64", "hpsi", "HF", "fcc2", "3x3x3", 5.0, "16x16x16", 4, 8, "fp64", tr=True),
        # HF exchange on 2x2x2 k, 10 Ha, 24^3: the library's plain configuration
        _case("hf_si2_24_apply_fp64", "apply", "HF", "fcc2", "2x2x2", 10.0, "24x24x24", 4, 12, "fp64"),
        # HF exchange on a production mesh and grid in mixed precision
        _case("hf_si2_36_apply_mixed", "apply", "HF", "fcc2", "3x3x3", 14.0, "36x36x36", 4, 12, "mixed"),
        # one SCF iteration's first apply of a TC run from host buffers: upload, per-state work, all TC terms
        _case("tc_si2_32_scf_mixed", "scf", "TC", "fcc2", "2x2x2", 10.0, "32x32x32", 4, 8, "mixed"),
        # a later Davidson apply of the same run in double precision (state resident)
        _case("tc_si2_32_apply_fp64", "apply", "TC", "fcc2", "2x2x2", 10.0, "32x32x32", 4, 8, "fp64"),
        # a small TC run reduced by time reversal, from host buffers
        _case("tc_si2_16_scf_fp64", "scf", "TC", "fcc2", "3x3x3", 4.0, "16x16x16", 4, 6, "fp64", tr=True),
        # spin-polarised TC with three different Jastrow channels on an uneven grid
        _case("tc_lsda_uneven_scf_fp64", "scf", "TC", "fcc2", "2x2x1", 6.0, "20x18x21", 4, 6, "fp64", nspin=2,
              channels="unequal"),
        # energy and its gradients for a Jastrow optimisation: electron gas, Gamma only
        _case("heg_40_gradient_fp64", "gradient", "BITC", "heg54", "1x1x1", 1.661, "40x40x40", 27, 27, "fp64"),
        # a Davidson apply of BITC in double precision (state resident)
        _case("bitc_si2_36_apply_fp64", "apply", "BITC", "fcc2", "2x2x2", 14.0, "36x36x36", 4, 8, "fp64"),
        # per-state work and apply of BITC on device buffers, 3x3x3 mesh: the largest pass here
        _case("bitc_si2_36_27k_step_mixed", "step", "BITC", "fcc2", "3x3x3", 14.0, "36x36x36", 4, 8, "mixed"),
        # eight-atom cube on 48^3: large plane-wave blocks, few k-points
        _case("tc_si8_48_step_mixed", "step", "TC", "sc8", "1x1x2", 20.0, "48x48x48", 16, 48, "mixed"),
        # the dense subspace step of block Davidson at the eight-atom cube's sizes
        _case("davidson_si8_fp64", "davidson", "TC", "sc8", "1x1x1", 20.0, "48x48x48", 16, 48, "fp64"),
    ]


# ------------------------------------------------------------- geometry --
def _lattice(cell):
    if cell == "fcc2":
        return (SI_A / 2.0) * np.array([[-1.0, 0.0, 1.0], [0.0, 1.0, 1.0], [-1.0, 1.0, 0.0]])
    if cell == "sc8":
        return SI_A * np.eye(3)
    # "heg54": 54 electrons at r_s = 2
    return np.cbrt(54 * FOURPI / 3.0 * 8.0) * np.eye(3)


def _dims(text):
    return tuple(int(x) for x in text.split("x"))


def _kpoints(case):
    """(irreducible k, has a time-reversed partner) of the Gamma-centred mesh."""
    mesh = _dims(case["mesh"])
    full = [np.array([i / mesh[0], j / mesh[1], k / mesh[2]])
            for i, j, k in itertools.product(range(mesh[0]), range(mesh[1]), range(mesh[2]))]
    if not case["tr"]:
        return [(k, False) for k in full]
    out, seen = [], set()
    for k in full:
        key, mkey = (tuple(np.round(np.mod(s * k, 1.0), 6) % 1.0) for s in (1, -1))
        if key in seen:
            continue
        seen.update((key, mkey))
        out.append((k, key != mkey))
    return out


def _sphere(recip, k, ecut, grid):
    """Miller indices of the plane waves 1/2 |k+G|^2 < ecut, by length."""
    ax = [np.arange(-((n - 1) // 2), n // 2 + 1) for n in grid]
    M = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    G = (k[None, :] + M) @ recip
    e = 0.5 * np.einsum("ij,ij->i", G, G)
    M, e = M[e < ecut], e[e < ecut]
    if np.any(np.abs(M) * 2 >= np.array(grid)[None, :]):
        raise ValueError("plane-wave sphere does not fit the FFT grid")
    return M[np.lexsort((M[:, 2], M[:, 1], M[:, 0], np.round(e, 12)))].astype(np.int64)


def _gindex(M, grid):
    w = np.mod(M, np.array(grid))
    return (w[:, 0] + grid[0] * (w[:, 1] + grid[1] * w[:, 2])).astype(np.int32)


def _orbitals(rng, M, kG2, nb, nspin, sym):
    """Seeded orthonormal bands with a decaying spectrum; `sym` closes them
    under time reversal (k-points that are their own partner)."""
    X = rng.standard_normal((nspin, len(M), nb)) + 1j * rng.standard_normal((nspin, len(M), nb))
    X *= np.exp(-kG2 / 8.0)[None, :, None]
    if sym is not None:
        X = 0.5 * (X + X[:, sym].conj())
    return [np.linalg.qr(x)[0] for x in X]


class _Problem:
    """Geometry, orbitals and density of one case, from the seed alone."""

    def __init__(self, case, seed):
        self.case = case
        self.grid = _dims(case["grid"])
        self.N = int(np.prod(self.grid))
        self.lattice = _lattice(case["cell"])
        self.recip = 2.0 * np.pi * np.linalg.inv(self.lattice).T
        self.omega = float(abs(np.linalg.det(self.lattice)))
        self.nspin = case["nspin"]
        self.method = case["method"]
        self.bitc = self.method == "BITC"
        self.nocc, self.nb = case["nocc"], case["nbands"]
        kp = _kpoints(case)
        self.kirr = [k for k, _ in kp]
        self.partner = [p for _, p in kp]
        self.kall = [(ik, s) for ik, p in enumerate(self.partner) for s in ((1, -1) if p else (1,))]
        self.nkpt = len(self.kall)
        if case["method"] == "HF":
            self.A, self.F = np.zeros((2, 2)), np.ones((2, 2))
        elif case["channels"] == "equal":
            self.A, self.F = np.full((2, 2), 0.5), np.full((2, 2), 1.2)
        else:
            self.A = np.full((2, 2), 0.5)
            self.F = np.array([[1.3, 1.0], [1.0, 1.2]])
        rng = np.random.default_rng([11, seed])
        self.M, self.kg, self.phi, self.chi = [], [], [], []
        for k in self.kirr:
            M = _sphere(self.recip, k, case["ecut"], self.grid)
            kg = (k[None, :] + M) @ self.recip
            g2 = np.einsum("ij,ij->i", kg, kg)
            sym = None
            if case["tr"] and np.allclose(2 * k, np.rint(2 * k)):
                pos = {tuple(m): i for i, m in enumerate(M)}
                shift = np.rint(-2 * k).astype(np.int64)
                sym = np.array([pos[tuple(shift - m)] for m in M])
            phi = _orbitals(rng, M, g2, self.nb, self.nspin, sym)
            self.M.append(M)
            self.kg.append(kg)
            self.phi.append(phi)
            if self.bitc:
                left = _orbitals(rng, M, g2, self.nb, self.nspin, sym)
                left = [0.3 * x + p for x, p in zip(left, phi)]
                self.chi.append([x @ np.linalg.inv(p.conj().T @ x) for x, p in zip(left, phi)])
            else:
                self.chi.append(phi)
        self.fillval = 2.0 if self.nspin == 1 else 1.0
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.density = self._density()

    # -- fields on the real-space grid ------------------------------------
    def gidx(self, ik, sign):
        return _gindex(sign * self.M[ik], self.grid)

    def to_r(self, coef, gidx):
        """coef [bands, npw] on grid indices gidx -> [bands, n2, n1, n0]."""
        n0, n1, n2 = self.grid
        g = torch.zeros((coef.shape[0], self.N), dtype=torch.complex128, device=self.dev)
        g[:, torch.as_tensor(gidx, dtype=torch.long, device=self.dev)] = coef
        return torch.fft.ifftn(g.view(-1, n2, n1, n0), dim=(1, 2, 3), norm="forward")

    def tensor(self, x):
        return torch.as_tensor(np.ascontiguousarray(x), device=self.dev)

    def orbital(self, s, ik, sign, nb, left=False):
        c = self.tensor((self.chi if left else self.phi)[ik][s][:, :nb].T)
        return c if sign > 0 else c.conj().resolve_conj()

    def _density(self):
        n0, n1, n2 = self.grid
        out = torch.zeros((2, n2, n1, n0), dtype=torch.complex128, device=self.dev)
        for s in range(self.nspin):
            for ik, sign in self.kall:
                gi = self.gidx(ik, sign)
                phi = self.to_r(self.orbital(s, ik, sign, self.nocc), gi)
                chi = self.to_r(self.orbital(s, ik, sign, self.nocc, True), gi) if self.bitc else phi
                out[s] += self.fillval * (chi.conj() * phi).sum(0)
        if self.nspin == 1:
            out[0] /= 2.0
            out[1] = out[0]
        return out

    # -- the library's containers -------------------------------------------
    def system(self):
        flat = lambda L: np.concatenate([np.ascontiguousarray(L[k][s].T).ravel() for s in range(self.nspin)
                                         for k in range(len(self.kirr))])
        gi = np.concatenate([self.gidx(ik, sg) for ik, sg in self.kall] * self.nspin)
        nk = len(self.kirr)
        filling = np.zeros((self.nspin, nk, self.nb))
        filling[:, :, :self.nocc] = self.fillval
        phik = flat(self.phi)
        s = TCSystem(
            nr=self.grid, recip=self.recip, lattice=self.lattice, omega=self.omega, method=self.method,
            nspin=self.nspin, nsym_k=np.array([2 if p else 1 for p in self.partner], dtype=np.int32),
            kvec=np.array([sg * self.kirr[ik] for ik, sg in self.kall]),
            time_rev=np.array([sg < 0 for _, sg in self.kall], dtype=np.uint8),
            rot_index=np.zeros(self.nkpt, dtype=np.int32), rotation=np.eye(3, dtype=np.int32)[None],
            translation=np.zeros((1, 3)), num_kpoints=self.nkpt,
            npw=np.array([len(m) for m in self.M], dtype=np.int32), gindex=gi,
            phase=np.ones(len(gi), dtype=np.complex128), jastrow_A=self.A, jastrow_F=self.F,
            includes_div_correction=True, alpha_Vaux=0.0, sum_Vaux=np.zeros(nk),
            nbands=np.full(self.nspin, self.nb, dtype=np.int32),
            nocc=np.full((self.nspin, nk), self.nocc, dtype=np.int32), filling=filling.ravel(), phik=phik,
            phik_left=flat(self.chi) if self.bitc else None,
            density=self.density.cpu().numpy().reshape(2, self.N),
            nb_apply=np.full((self.nspin, nk), self.nb, dtype=np.int32), psi=phik.copy())
        s.alpha_Vaux, s.sum_Vaux = sum_of_vaux(s)
        return s

    def pseudo(self):
        """A two-projector pseudopotential (l = 0 and 1) on both atoms and a
        smooth local potential."""
        rng = np.random.default_rng(5)
        d = rng.standard_normal(2)
        rad = rng.uniform(0.5, 1.5, 2)
        proj = []
        for kg in self.kg:
            q = np.linalg.norm(kg, axis=1)
            rows = [np.exp(-rad[0] * q ** 2 / 4) / np.sqrt(FOURPI) + 0j]
            f1 = np.sqrt(3.0 / FOURPI) * np.exp(-rad[1] * q ** 2 / 4)
            rows += [-1j * f1 * kg[:, x] for x in range(3)]
            proj.append(np.stack(rows))
        n0, n1, n2 = self.grid
        z, y, x = np.meshgrid(np.arange(n2) / n2, np.arange(n1) / n1, np.arange(n0) / n0, indexing="ij")
        vloc = np.zeros_like(x)
        for _ in range(4):
            h = rng.integers(-2, 3, size=3)
            vloc += rng.standard_normal() * np.cos(2 * np.pi * (h[0] * x + h[1] * y + h[2] * z))
        pos = np.array([[0.0, 0.0, 0.0], [0.25, 0.25, 0.25]]) @ self.lattice
        pp = Pseudo(vloc=vloc.ravel(), species_of_atom=np.zeros(2, dtype=np.int32), atom_pos=pos, lbeta=[[0, 1]],
                    dij=[np.diag(d)], projector=np.concatenate([p.ravel() for p in proj]))
        return pp, proj, np.array([d[0], d[1], d[1], d[1]])


# --------------------------------------------------------------- passes --
def prepare(case, seed):
    if case["kind"] == "davidson":
        return _prepare_davidson(case, seed)
    P = _Problem(case, seed)
    system = P.system()
    ctx = Context(system, case["precision"])
    st = dict(case=case, kind=case["kind"], ctx=ctx, system=system, terms=H2_BITS[P.method] | H3_BITS[P.method])
    if case["kind"] == "hpsi":
        ctx.set_pseudo(P.pseudo()[0])
    if case["kind"] != "scf":
        ctx.set_state()
    if case["kind"] in ("apply", "step"):
        st["stream"] = torch.cuda.ExternalStream(int(ctx.stream))
        st["psi"] = torch.from_numpy(system.psi).cuda()
        st["h2"] = torch.zeros_like(st["psi"])
        st["h3"] = torch.zeros_like(st["psi"])
    elif case["kind"] == "gradient":
        st["dchi"] = torch.zeros(system.phik.size, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    return st


def run(state):
    kind = state["kind"]
    if kind == "davidson":
        return _run_davidson(state)
    ctx, terms = state["ctx"], state["terms"]
    if kind == "hpsi":                           # H1 psi and H2 psi of a block, host buffers
        h1 = ctx.apply_h1(abi.TERMS_H1)
        h2, _ = ctx.apply(terms)
        return h1, h2
    if kind == "scf":                            # a new SCF iteration's orbitals, then the first block
        ctx.set_state()
        return ctx.apply(terms)
    if kind == "gradient":
        e2, e3, du, dv = ctx.energy_grad(abi.TERMS_TC, dchi_ptr=state["dchi"].data_ptr(), tables=True)
        return np.array([e2, e3]), state["dchi"], du, dv
    if kind == "step":                           # device buffers, per-state work included
        ctx.refresh_state()
    h3 = 0 if ctx.system.method == "HF" else state["h3"].data_ptr()
    with torch.cuda.stream(state["stream"]):     # the library's stream: zeroed before the terms are added
        state["h2"].zero_()
        if h3:
            state["h3"].zero_()
    ctx.apply_device(terms, state["psi"].data_ptr(), state["h2"].data_ptr(), h3)
    return (state["h2"], state["h3"]) if h3 else state["h2"]


def _davidson_inputs(case, seed):
    """Orthonormal basis of one k-point, the operator applied to it, and a second
    basis of twice the size for the Rayleigh-Ritz step."""
    recip = 2.0 * np.pi * np.linalg.inv(_lattice(case["cell"])).T
    k = np.array([0.1, 0.2, 0.3])
    M = _sphere(recip, k, case["ecut"], _dims(case["grid"]))
    kg = (k[None, :] + M) @ recip
    kg2 = np.einsum("ij,ij->i", kg, kg)
    npw, nb = len(M), case["nbands"]
    rng = np.random.default_rng([13, seed])
    rnd = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)
    env = np.exp(-kg2 / 16.0)[:, None]
    B = np.linalg.qr(rnd(npw, 2 * nb) * env)[0]
    # H1 = kinetic; H2, H3 = low-rank non-Hermitian parts with a decaying spectrum
    U2, W2, U3, W3 = (rnd(npw, 16) * env / math.sqrt(npw) for _ in range(4))
    H = [0.5 * kg2[:, None] * B, -3.0 * U2 @ (U2.conj().T @ B) + 0.3 * U2 @ (W2.conj().T @ B),
         0.5 * U3 @ (W3.conj().T @ B)]
    eig = np.einsum("ij,ij->j", B.conj(), H[0] + H[1] + H[2])[:nb] * (1.0 + 0.01 * rng.standard_normal(nb))
    return dict(npw=npw, nb=nb, kg2=kg2, B=B, H=H, eig=eig)


def _prepare_davidson(case, seed):
    d = _davidson_inputs(case, seed)
    rows = lambda X: torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    nb = d["nb"]
    V = torch.zeros((2 * nb, d["npw"]), dtype=torch.complex128, device="cuda")
    V[:nb] = rows(d["B"][:, :nb])
    st = dict(kind="davidson", case=case, nb=nb, V=V, basis=rows(d["B"]), HB=[rows(h) for h in d["H"]],
              phi=V[:nb].clone(), Hphi=[rows(h[:, :nb]) for h in d["H"]], kg2=torch.from_numpy(d["kg2"]).cuda(),
              eig=d["eig"])
    torch.cuda.synchronize()
    return st


def _run_davidson(st):
    """Expansion of the basis by the preconditioned residuals, then the
    Rayleigh-Ritz step of a full basis and the orthonormalised Ritz vectors."""
    nb = st["nb"]
    n = davidson_expand(st["V"], nb, st["phi"], st["Hphi"], st["kg2"], st["eig"])
    w, e, vo, _ = subspace_ritz(st["basis"], st["HB"], nb)
    vo = vo.contiguous()
    gram_schmidt(vo)
    return dict(rows=n, V=st["V"], eigenvalues=w, energies=e, ritz=vo)


# ---------------------------------------------------- plain torch numbers --
def _uk(G2, A, F):
    if A == 0.0:
        return torch.zeros_like(G2)
    z = G2 < 1e-12
    g = torch.where(z, torch.ones_like(G2), G2)
    return torch.where(z, torch.full_like(G2, -FOURPI * A * F * F), FOURPI * A / (g * (g * F * F + 1.0)))


def _v2body(G2, A, F):
    z = G2 < 1e-12
    g2 = torch.where(z, torch.ones_like(G2), G2)
    g, f2 = torch.sqrt(g2), F * F * g2
    v = (FOURPI / g2 - FOURPI * A / (1.0 + f2)
         + (math.pi * A * A / (F * F) / g) * (math.pi * f2 + (4 + 2 * f2) * torch.atan(F * g / 2)
                                              - (4 + 4 * f2) * torch.atan(F * g)))
    return torch.where(z, torch.full_like(G2, -2.0 * math.pi * A * A / F), v)


class _Exact:
    """The operator terms of a problem in plain torch, complex128: every pair
    sum written out on the full grid."""

    def __init__(self, P, nb_apply, sumv, alpha, hartree=True):
        self.P, self.nb, self.hartree = P, nb_apply, hartree
        self.sumv, self.alpha = sumv, alpha
        n0, n1, n2 = P.grid
        ax = [torch.arange(n, device=P.dev) for n in (n2, n1, n0)]
        ax = [torch.where(a <= n // 2, a, a - n).to(torch.float64) for a, n in zip(ax, (n2, n1, n0))]
        m2, m1, m0 = torch.meshgrid(*ax, indexing="ij")
        b = P.recip
        self.G = torch.stack([m0 * b[0, d] + m1 * b[1, d] + m2 * b[2, d] for d in range(3)])
        self.G2 = (self.G ** 2).sum(0)
        self.nk, self.om = P.nkpt, P.omega
        self.occ = {}
        for s in range(P.nspin):
            for a, (ik, sg) in enumerate(P.kall):
                gi = P.gidx(ik, sg)
                c = P.orbital(s, ik, sg, P.nocc)
                kg = P.tensor(sg * P.kg[ik])
                phi = P.to_r(c, gi)
                grad = torch.stack([P.to_r(c * kg[:, d], gi) for d in range(3)], 1)
                chi = P.to_r(P.orbital(s, ik, sg, P.nocc, True), gi) if P.bitc else phi
                self.occ[s, a] = (phi, chi, grad)

    fwd = staticmethod(lambda x: torch.fft.fftn(x, dim=(-3, -2, -1), norm="forward"))
    inv = staticmethod(lambda x: torch.fft.ifftn(x, dim=(-3, -2, -1), norm="forward"))

    def kq(self, k, a):
        ik, sg = self.P.kall[a]
        q = torch.as_tensor((np.asarray(k) - sg * self.P.kirr[ik]) @ self.P.recip, device=self.P.dev)
        K = self.G + q[:, None, None, None]
        return K, (K ** 2).sum(0)

    def gather(self, acc, ik):
        idx = torch.as_tensor(self.P.gidx(ik, 1), dtype=torch.long, device=self.P.dev)
        return self.fwd(acc).reshape(-1)[idx]

    def div2(self, s, ik, psi):
        """h of the G = 0 correction: sum_b f dc <chi_b|psi> phi_b."""
        P = self.P
        dc = -(1.0 / math.sqrt(math.pi * self.alpha) - self.sumv[ik] / (self.nk * self.om))
        if P.nspin == 1:
            dc /= 2.0
        phi, chi = P.orbital(s, ik, 1, P.nocc), P.orbital(s, ik, 1, P.nocc, True)
        return P.fillval * dc * ((chi.conj() @ psi) @ phi)

    def local(self):
        """Per-state fields: densities in G, dnu, Hartree and local three-body potentials."""
        P = self.P
        ns = P.nspin
        n = P.density
        self.nG = self.fwd(n)
        if P.method == "HF":
            g2 = torch.where(self.G2 < 1e-12, torch.ones_like(self.G2), self.G2)
            self.vh = self.inv(torch.where(self.G2 < 1e-12, torch.zeros_like(g2), FOURPI / g2) * self.nG.sum(0))
            return
        u = {(a, b): _uk(self.G2, P.A[a, b], P.F[a, b]) for a in range(2) for b in range(2)}
        self.u = u
        self.dnu = [self.inv(sum(u[s, j] * self.nG[j] for j in range(2)) * self.G) for s in range(ns)]
        W = [self.fwd(self.dnu[s] * n[s]) for s in range(ns)]
        self.v3a1 = [(self.dnu[s] ** 2).sum(0) for s in range(ns)]
        self.v3b1 = [self.inv(sum(u[s, t] * (self.G * W[0 if ns == 1 else t]).sum(0) for t in range(2)))
                     for s in range(ns)]
        pg = []
        for s in range(ns):
            t = sum(P.fillval * (chi.conj()[:, None] * grad).sum(0)
                    for (phi, chi, grad) in (self.occ[s, a] for a in range(self.nk)))
            pg.append(self.fwd(t))
        sf = 2.0 if ns == 1 else 1.0
        self.v2h = [self.inv(sum(_v2body(self.G2, P.A[s, j], P.F[s, j]) * self.nG[j]
                                 + u[s, j] * (self.G * pg[0 if ns == 1 else j]).sum(0) / sf for j in range(2)))
                    for s in range(ns)]

    def occupied_pairs(self):
        """Intermediates of tc3a2a4b2b5: 3a2 / 3b2 potentials and the rotated Q, B fields."""
        P = self.P
        ns, dev = P.nspin, P.dev
        zero = lambda *s: torch.zeros(s + self.G2.shape, dtype=torch.complex128, device=dev)
        self.v3a2, self.v3b2 = zero(ns), zero(ns)
        self.Qt, self.Bt = {}, {}
        f = P.fillval
        first = {}
        for a, (ik, sg) in enumerate(P.kall):
            if sg > 0:
                first[ik] = a
        for sq in range(ns):
            q3b2 = zero(3)
            for ik, k in enumerate(P.kirr):
                phi2, chi2, _ = self.occ[sq, first[ik]]
                T, Q, B = zero(P.nocc, ns), zero(P.nocc, 3), zero(P.nocc, 3)
                for a in range(self.nk):
                    phi1, chi1, _ = self.occ[sq, a]
                    K, K2 = self.kq(k, a)
                    us = [_uk(K2, P.A[sq, x], P.F[sq, x]) for x in range(2)]
                    for i2 in range(P.nocc):
                        pp = self.fwd(chi1.conj() * phi2[i2])
                        pj = self.fwd(phi1.conj() * chi2[i2]) if P.bitc else None
                        for x in range(2):
                            o1 = self.inv(pp[:, None] * (K * us[x]))
                            o2 = self.inv(pj[:, None] * (K * us[x])) if P.bitc else o1
                            T[i2, 0 if ns == 1 else x] -= f * (o2.conj() * o1).sum((0, 1))
                            if x == sq:
                                Q[i2] += f * (o1 * phi1[:, None]).sum(0)
                                B[i2] -= f * (o2.conj() * chi1.conj()[:, None]).sum(0)
                if not P.bitc:
                    B = -Q.conj()
                T = self.fwd(T)
                dcorr = self.nk * self.om / math.sqrt(math.pi * self.alpha) - self.sumv[ik]
                pp = self.fwd(chi2.conj()[:, None] * phi2[None, :])          # [i1][i2]
                pj = self.fwd(chi2.conj()[None, :] * phi2[:, None])
                for x in range(2):
                    Ax, Fx = P.A[sq, x], P.F[sq, x]
                    c = FOURPI * Ax * f
                    d = c * _uk(self.G2, Ax, Fx) * (pp * pj[..., :1, :1, :1] + pp[..., :1, :1, :1] * pj)
                    d[..., 0, 0, 0] = c * (Ax * dcorr - FOURPI * Ax * Fx * Fx) * pp[..., 0, 0, 0] * pj[..., 0, 0, 0]
                    T[:, 0 if ns == 1 else x] -= d.sum(0)
                Tr = self.inv(T)
                for a, (jk, sg) in enumerate(P.kall):
                    if jk != ik:
                        continue
                    Qa, Ba = (Q, B) if sg > 0 else (-Q.conj(), -B.conj())
                    self.v3a2 += f * (Tr if sg > 0 else Tr.conj()).sum(0)
                    self.Qt[sq, a], self.Bt[sq, a] = Qa, Ba
                    q3b2 += f * (Ba * self.occ[sq, a][0][:, None]).sum(0)
            qG = (self.G * self.fwd(q3b2)).sum(0)
            for s in range(ns):
                up = self.u[s, 0] + self.u[s, 1] if ns == 1 else self.u[s, sq]
                self.v3b2[s] += self.inv(up * qG)

    def band(self, s, ik, psi):
        """(H2 psi, H3 psi) of one trial orbital psi [npw] at irreducible k."""
        P = self.P
        ns, f, k = P.nspin, P.fillval, P.kirr[ik]
        Nk, Om = self.nk, self.om
        gi = P.gidx(ik, 1)
        kg = P.tensor(P.kg[ik])
        r = P.to_r(psi[None], gi)[0]
        half = 2.0 if ns == 1 else 1.0
        if P.method == "HF":
            acc = torch.zeros_like(r)
            for a in range(self.nk):
                phi = self.occ[s, a][0]
                _, K2 = self.kq(k, a)
                v = torch.where(K2 < 1e-8, torch.zeros_like(K2), 1.0 / torch.where(K2 < 1e-8, torch.ones_like(K2), K2))
                acc += f * (phi * self.inv(v * self.fwd(phi.conj() * r))).sum(0)
            h2 = self.gather(acc * (-FOURPI / (Nk * Om) / half) + self.vh * r / (Nk * Om), ik)
            return h2 + self.div2(s, ik, psi), None
        g = torch.stack([P.to_r((psi * kg[:, d])[None], gi)[0] for d in range(3)])
        base = 1.0 / (Nk * Om) ** 2
        a3, b3, b4, b6 = -base, base, -base, base
        fa2, fb2, fa4 = -0.5 * base, base, base
        if ns == 1:
            a3, b3, b4, b6 = a3 / 2, b3 / 2, b4 / 4, b6 / 2
            fa2, fb2, fa4 = fa2 / 4, fb2 / 4, fa4 / 4
        acc2 = torch.zeros_like(r)
        dn = self.dnu[s]
        acc3 = (0.5 * base * self.v3a1[s] - base * self.v3b1[s] + fa2 * self.v3a2[s] + fb2 * self.v3b2[s]) * r
        qsum = torch.zeros_like(dn)
        dnp = dn * r
        tables = []
        for a in range(self.nk):
            phi, chi, grad = self.occ[s, a]
            K, K2 = self.kq(k, a)
            u = [_uk(K2, P.A[x, s], P.F[x, s]) for x in range(2)]
            du = K * u[s]
            tables.append(du)
            cc = chi.conj()
            rho = self.fwd(cc * r)
            o = _v2body(K2, P.A[s, s], P.F[s, s]) * rho + (self.fwd(cc[:, None] * g) * du).sum(1)
            w = self.inv(rho[:, None] * du)
            acc2 += f * (phi * self.inv(o) - (grad * w).sum(1)).sum(0)
            qsum += f * (phi[:, None] * w).sum(0)
            acc3 += f * fa4 * (self.Qt[s, a] * w).sum((0, 1))
            e = b3 * (self.fwd(cc[:, None] * dnp) * du).sum(1) - fa4 * (self.fwd(self.Bt[s, a] * r) * du).sum(1)
            for x in range(2):
                wx = w if x == s else self.inv(rho[:, None] * (K * u[x]))
                e = e + b6 * (self.fwd(P.density[x] * wx) * (K * u[x])).sum(1)
            acc3 += f * (phi * self.inv(e)).sum(0)
        acc3 += a3 * (qsum * dn).sum(0)
        for a in range(self.nk):
            phi, chi, _ = self.occ[s, a]
            acc3 += b4 * f * (phi * self.inv((self.fwd(chi.conj()[:, None] * qsum) * tables[a]).sum(1))).sum(0)
        # G = 0 correction of 3b6
        tG = sum(FOURPI * self.nG[j] * P.A[0, int(j != s)] * _uk(self.G2, P.A[0, int(j != s)], P.F[0, int(j != s)])
                 for j in range(2))
        tG[0, 0, 0] = 0.0
        tR = self.inv(tG)
        dcorr = Nk * Om / math.sqrt(math.pi * self.alpha) - self.sumv[ik]
        t1 = sum(FOURPI * (dcorr * P.A[s, j] - FOURPI * P.A[s, j] * P.F[s, j] ** 2) * P.A[s, j] * self.nG[j, 0, 0, 0]
                 for j in range(2))
        pg, cg = P.orbital(s, ik, 1, P.nocc), P.orbital(s, ik, 1, P.nocc, True)
        a0 = next(a for a, (jk, sg) in enumerate(P.kall) if jk == ik and sg > 0)
        phi, chi, _ = self.occ[s, a0]
        cpi = cg.conj() @ psi
        dot2 = (chi.conj() * r * tR).mean((1, 2, 3))
        acc3 += f * b6 * tR * (cpi[:, None, None, None] * phi).sum(0)
        h3 = self.gather(acc3, ik) + f * b6 * ((t1 * cpi + dot2) @ pg)
        acc2 = -acc2 / (Nk * Om) / half
        if self.hartree:
            acc2 = acc2 + (self.v2h[s] * r - (dn * g).sum(0)) / (Nk * Om)
        return self.gather(acc2, ik) + self.div2(s, ik, psi), h3

    def apply(self):
        P = self.P
        self.local()
        if P.method != "HF":
            self.occupied_pairs()
        h2, h3 = [], []
        for s in range(P.nspin):
            for ik in range(len(P.kirr)):
                c = P.orbital(s, ik, 1, self.nb)
                for b in range(self.nb):
                    x, y = self.band(s, ik, c[b])
                    h2.append(x)
                    h3.append(y)
        h2 = torch.cat(h2)
        return h2, (None if P.method == "HF" else torch.cat(h3))


def _exact_gradient(P, X):
    """E2, E3, dE/d conj(chi) and the two-body Jastrow-table gradients (Gamma only, one spin)."""
    h2, h3 = X.apply()
    npw, no, f, Nk = len(P.M[0]), P.nocc, P.fillval, X.nk
    h2, h3 = h2.view(no, npw), h3.view(no, npw)
    chi = P.orbital(0, 0, 1, no, True)
    e = np.array([complex(f * (chi.conj() * h).sum() / (n * Nk)) for h, n in ((h2, 2), (h3, 3))])
    dchi = torch.zeros((P.nb, npw), dtype=torch.complex128, device=P.dev)
    dchi[:no] = f / Nk * (h2 + h3)
    phi, ch, grad = X.occ[0, 0]
    cf = -1.0 / (Nk * X.om) / 2.0 / (2.0 * Nk) * f * f
    neg = lambda g: torch.roll(torch.flip(g, (-3, -2, -1)), (1, 1, 1), (-3, -2, -1))
    dv, du = torch.zeros_like(X.nG[0]), torch.zeros_like(X.nG[0])
    for i in range(no):
        rij = X.fwd(ch[i].conj() * phi)                       # rho_ij, all j
        rji = neg(X.fwd(ch.conj() * phi[i]))                  # rho_ji(-G)
        gij = X.fwd(ch[i].conj() * grad)
        gji = neg(X.fwd(ch.conj()[:, None] * grad[i][None]))
        dv += cf * (rij * rji).sum(0)
        du += cf * (X.G * (gij * rji[:, None] - rij[:, None] * gji).sum(0)).sum(0)
    return e, dchi.reshape(-1), du.reshape(1, -1).cpu().numpy(), dv.reshape(1, -1).cpu().numpy()


def _exact_h1(P, nb):
    _, proj, d = P.pseudo()
    pp = P.pseudo()[0]
    n0, n1, n2 = P.grid
    v = P.tensor(pp.vloc.reshape(n2, n1, n0))
    out = []
    for s in range(P.nspin):
        for ik in range(len(P.kirr)):
            c = P.orbital(s, ik, 1, nb)
            kg = P.tensor(P.kg[ik])
            h = 0.5 * (kg ** 2).sum(1) * c
            G = P.M[ik] @ P.recip
            for pos in pp.atom_pos:
                B = P.tensor(np.exp(1j * (G @ pos))[None, :] * proj[ik])
                h = h + (c @ B.T * P.tensor(d)) @ B.conj()
            idx = torch.as_tensor(P.gidx(ik, 1), dtype=torch.long, device=P.dev)
            r = torch.fft.fftn(v * P.to_r(c, P.gidx(ik, 1)), dim=(1, 2, 3), norm="forward")
            out.append((h + r.reshape(nb, -1)[:, idx]).reshape(-1))
    return torch.cat(out)


def _exact_davidson(case, seed):
    d = _davidson_inputs(case, seed)
    nb, kg2 = d["nb"], d["kg2"]
    V = [d["B"][:, j].copy() for j in range(nb)]
    Hs = d["H"][0] + d["H"][1] + d["H"][2]
    rows = nb
    for b in range(nb):
        p = d["B"][:, b]
        x = kg2 / (np.sum(kg2 * np.abs(p) ** 2) / np.sum(np.abs(p) ** 2))
        poly = 27 + x * (18 + x * (12 + 8 * x))
        t = -(poly / (poly + 16 * x ** 4)) * (Hs[:, b] - d["eig"][b] * p)
        t /= np.linalg.norm(t)
        for v in V:
            t = t - np.vdot(v, t) * v
        V.append(t / np.linalg.norm(t))
        rows += 1
    Hn = [d["B"].conj().T @ h for h in d["H"]]
    w, X = np.linalg.eig(Hn[0] + Hn[1] + Hn[2])
    order = np.argsort(w.real, kind="stable")
    X = X[:, order][:, :nb]
    X = X / np.linalg.norm(X, axis=0)
    en = np.stack([np.einsum("ai,ab,bi->i", X.conj(), h, X) for h in Hn])
    return dict(rows=rows, V=np.stack(V), eigenvalues=w[order], energies=en, ritz=None)


def exact(case, seed):
    """What run() returns, in plain torch / numpy with 64-bit numbers."""
    if case["kind"] == "davidson":
        return _exact_davidson(case, seed)
    P = _Problem(case, seed)
    system = P.system()
    nb = P.nocc if case["kind"] == "gradient" else P.nb
    X = _Exact(P, nb, system.sum_Vaux, system.alpha_Vaux, hartree=case["kind"] != "gradient")
    if case["kind"] == "gradient":
        return _exact_gradient(P, X)
    h2, h3 = X.apply()
    if case["kind"] == "hpsi":
        return _exact_h1(P, nb), h2
    if P.method == "HF":
        return (h2, torch.zeros_like(h2)) if case["kind"] == "scf" else h2
    return h2, h3


# ----------------------------------------------------------------- sizes --
def _counts(case):
    lat = _lattice(case["cell"])
    recip = 2.0 * np.pi * np.linalg.inv(lat).T
    omega = abs(np.linalg.det(lat))
    R = math.sqrt(2.0 * case["ecut"])
    npw = FOURPI / 3.0 * R ** 3 * omega / (2.0 * np.pi) ** 3
    kp = _kpoints(case)
    nk, nk_all = len(kp), sum(2 if p else 1 for _, p in kp)
    # points of a grid whose periodic images of the pair-density sphere (radius 2 R) stay apart
    b = min(np.linalg.norm(np.array(m) @ recip) for m in itertools.product((-1, 0, 1), repeat=3) if any(m))
    n = [min(g, math.ceil(4.0 * R / b)) for g in _dims(case["grid"])]
    return npw, nk, nk_all, float(np.prod(n))


def work(case):
    """Inputs read once and outputs written once; the pair transforms (on a grid
    that just holds the pair densities) at 5 P log2 P."""
    npw, nk, nk_all, pts = _counts(case)
    nb, no, ns = case["nbands"], case["nocc"], case["nspin"]
    if case["kind"] == "davidson":
        n2 = 2 * nb
        io = 16.0 * npw * (nb * 5 + n2 * 4 + 2 * nb)
        gs = 8.0 * 2 * npw * (nb * nb + 2 * nb * (nb - 1) / 2)
        return dict(bytes=io, flops=gs + 8.0 * npw * (3 * n2 * n2 + n2 * nb) + 25.0 * 8 * n2 ** 3)
    bands = ns * nk * nb
    blocks = 2 if case["method"] == "HF" else 3
    if case["kind"] == "hpsi":
        blocks = 4
    io = 16.0 * npw * (bands * blocks + ns * nk * no * (2 if case["method"] == "BITC" else 1))
    tgt = ns * nk * (no if case["kind"] == "gradient" else nb)
    src = nk_all * no
    fft = 5.0 * pts * math.log2(pts)
    flops = tgt * src * (2 if case["method"] == "HF" else 16) * fft
    if case["kind"] in ("scf", "step", "gradient") and case["method"] != "HF":
        flops += ns * nk * no * src * (8 if case["method"] == "BITC" else 4) * fft
    return dict(bytes=io, flops=flops)


_SIZES = (12, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32, 36, 40, 42, 45, 48)
_FAST = (12, 16, 24, 32, 36, 40, 48)


def _cost(case):
    """Rough relative cost of a pass, to keep drawn cases below the largest listed one."""
    w = work(case)
    _, _, _, pts = _counts(case)
    n = _dims(case["grid"])
    c = w["flops"] * np.prod(n) / pts
    if case["precision"] == "fp64":
        c *= 2.0
    if not (n[0] == n[1] == n[2] and n[0] in _FAST):
        c *= 6.0
    if case["channels"] == "unequal":
        c *= 2.0
    return c


def draw(rng):
    """One more case of the listed ranges."""
    limit = 0.8 * _cost(next(c for c in listed() if c["name"] == "bitc_si2_36_27k_step_mixed"))
    while True:
        kind = rng.choice(["apply", "apply", "step", "scf", "scf", "hpsi", "davidson", "gradient"])
        if kind == "davidson":
            c = _case("", kind, "TC", "sc8", "1x1x1", round(math.exp(rng.uniform(math.log(6.0), math.log(20.0))), 2),
                      "48x48x48", 8, rng.randint(4, 48), "fp64")
            c.pop("name")
            return c
        cell = rng.choice(["fcc2", "fcc2", "fcc2", "sc8"])
        method = "HF" if kind == "hpsi" else rng.choice(["TC", "BITC"] if kind == "gradient" else ["HF", "TC", "BITC"])
        if kind == "gradient":
            cell, mesh, tr = rng.choice(["heg54", "fcc2"]), "1x1x1", False
        else:
            top = 3 if cell == "fcc2" else 2
            mesh = "x".join(str(rng.randint(1, top)) for _ in range(3))
            tr = rng.random() < 0.25
        lo, hi = {"fcc2": (3.0, 14.0), "sc8": (3.0, 20.0), "heg54": (1.0, 2.5)}[cell]
        ecut = round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 2)
        lat = _lattice(cell)
        ext = math.sqrt(2.0 * ecut) * np.linalg.norm(lat, axis=1) / (2.0 * np.pi)
        # grids from one that holds the density of the sphere up to half as fine again
        n = []
        over = rng.uniform(1.0, 1.5)
        for e in ext:
            need = max(12, min(48, math.ceil((4.0 * e + 1) * over)))
            n.append(next(s for s in _SIZES if s >= need))
        if rng.random() < 0.2 and kind != "gradient":
            i = rng.randrange(3)
            j = _SIZES.index(n[i])
            n[i] = _SIZES[min(len(_SIZES) - 1, j + 1)]
        nocc = rng.randint(1, 4) if cell == "fcc2" else rng.randint(2, 16)
        nocc = rng.choice([14, 19, 27]) if cell == "heg54" else nocc
        nb = nocc + (0 if kind == "gradient" else rng.randint(0, 2 * nocc))
        nspin = 2 if kind in ("apply", "scf", "hpsi") and rng.random() < 0.25 else 1
        c = _case("", kind, method, cell, mesh, ecut, "x".join(map(str, n)), nocc, nb,
                  "fp64" if kind in ("hpsi", "gradient") or rng.random() < 0.5 else "mixed", nspin=nspin, tr=tr,
                  channels="unequal" if nspin == 2 and method != "HF" and rng.random() < 0.5 else "equal")
        c.pop("name")
        if _cost(c) > limit:
            continue
        try:
            recip = 2.0 * np.pi * np.linalg.inv(lat).T
            for k, _ in _kpoints(c):
                if len(_sphere(recip, k, ecut, n)) < 2 * nb:
                    raise ValueError("too few plane waves")
        except ValueError:
            continue
        return c

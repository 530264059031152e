"""The pass kernels at the sizes where they differ, and the choice of the work
grid, against the oracle.

- every compiled cubic size and run-time shape (uneven grids, cubic sizes without
  kernels of their own, lengths only the generic passes take), with a cutoff so
  large for the grid that the library has to work on the grid itself;
- the smaller work grid: HF where the pair densities wrap around its box, time
  reversal with k-differences beyond the first cell, TC with a density that is not
  band limited (the grid of the caller has to be used) and back, density output;
- the on-chip hf2x at each of its sizes, with several partial sums per target.

Tolerances as in test_gpu_parity.py: FP64 relative 1e-10, mixed 2e-5.
"""
import dataclasses

import numpy as np
import pytest

from tc_b200 import abi, synth
from tc_b200 import TCError
from tc_b200.context import Context
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "mixed": 2e-5}


def rel(a, b):
    d, m = np.abs(a - b).max(), np.abs(b).max()
    return d / m if m > 0 else d


def check(s, mask, prec, edge=None):
    """apply against the oracle; edge: the work grid's"""
    r2, r3 = O.apply(s, mask)
    with Context(s, prec) as ctx:
        ctx.set_state()
        g2, g3 = ctx.apply(mask)
        if edge:
            assert ctx.work_grid() == (edge,) * 3
    assert rel(g2, r2) < TOL[prec]
    if mask & ~abi.TERMS_H2:
        assert rel(g3, r3) < TOL[prec]


def tight(n, frac=0.21):
    """cutoff of an fcc Si sphere whose radius is `frac` times the shortest period of
    the n^3 grid: products of three-body terms fold onto the used components"""
    b = np.sqrt(3.0) * 2.0 * np.pi / 10.26
    return 0.5 * (frac * n * b) ** 2


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48])
def test_compiled_sizes(n, prec):
    s = synth.small("BITC", nr=(n, n, n), nk=1, ecut=tight(n), nbands=2, nocc=1, seed=n)
    check(s, abi.TERMS_TC, prec)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nr", [(21, 21, 21), (14, 14, 14), (20, 18, 21), (12, 25, 16), (35, 18, 20), (28, 42, 15),
                                (22, 20, 18), (26, 26, 26)])
def test_run_time_shapes(nr, prec):
    n = min(nr)
    s = synth.small("TC", nr=nr, nk=1, ecut=tight(n, 0.19), nbands=2, nocc=2, seed=n)
    check(s, abi.TERMS_TC, prec)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_run_time_shape_spin_channels(prec):
    """unequal Jastrow channels: the separate passes, both branches of x2"""
    s = synth.small("BITC", nr=(15, 18, 14), nk=1, ecut=2.5, nbands=2, nocc=1, nspin=2, F=np.array([[1.3, 1.0], [1.0, 1.2]]))
    check(s, abi.TERMS_TC, prec)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,ecut", [(12, 4.0), (15, 7.0), (16, 7.9), (18, 10.0), (20, 12.0)])
def test_on_chip_exchange(n, ecut, prec):
    """hf2x work grids of n^3 inside a finer grid; 16 sources.  On chip up to 20^3, in
    FP64 up to 18^3; 15^3 gives way to 16^3"""
    s = synth.small("HF", nr=(36, 36, 36), nk=2, ecut=ecut, nbands=3, nocc=2, seed=n)
    check(s, abi.TERM_HF2X, prec, 16 if n == 15 else n)
    with Context(s, prec) as ctx:
        ctx.set_state()
        ctx.profile(True)
        ctx.apply(abi.TERM_HF2X)
        assert ("hf2x:cube" in ctx.profile_read()) == (prec == "mixed" or n <= 18)


@pytest.mark.parametrize("prec,n,ecut", [("mixed", 20, 12.0), ("fp64", 18, 10.0)])
@pytest.mark.parametrize("budget", [1 << 20, 8 << 20])
def test_exchange_within_the_budget(budget, prec, n, ecut):
    """hf2x with a small budget of temporaries (1 MB: its kernel table does not fit and
    the passes run; 8 MB: on chip, targets in parts): results, and the device memory
    that an apply adds.  Besides twice the budget (temporaries and table) these are
    the orbitals on the grid, the accumulators, psi and h2, and 8 MB of small
    allocations; the partial sums alone were 47 MB in FP64 and 65 MB in mixed precision."""
    import torch
    s = synth.small("HF", nr=(36, 36, 36), nk=2, ecut=ecut, nbands=8, nocc=4, seed=n)
    r2, _ = O.apply(s, abi.TERM_HF2X)
    nt = 8 * 8
    rest = nt * n ** 3 * (16 + (16 if prec == "fp64" else 8)) + 2 * s.psi.nbytes + (8 << 20)
    for _ in range(2):                                     # the first loads the kernels
        with Context(s, prec, tmp_budget=budget) as ctx:
            ctx.set_state()
            assert ctx.work_grid() == (n,) * 3
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            g2, _ = ctx.apply(abi.TERM_HF2X)
            grown = free - torch.cuda.mem_get_info()[0]
            ctx.profile(True)
            ctx.apply(abi.TERM_HF2X)
            tags = set(ctx.profile_read())
        assert rel(g2, r2) < TOL[prec]
    assert ("hf2x:cube" in tags) == (budget > 1 << 20)
    assert grown <= 2 * budget + rest


def test_rotations_within_the_budget():
    """tc3a2a4b2b5 with scratch for one rotated orbital at a time"""
    s = synth.small("BITC", nr=(12, 12, 12), tr=True, ecut=2.5, nbands=2, nocc=2)
    r2, r3 = O.apply(s, abi.TERMS_TC)
    with Context(s, "fp64", tmp_budget=1 << 18) as ctx:
        ctx.set_state()
        g2, g3 = ctx.apply(abi.TERMS_TC)
    assert rel(g2, r2) < TOL["fp64"]
    assert rel(g3, r3) < TOL["fp64"]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", ["HF", "TC"])
def test_work_grid_time_reversal(method, prec):
    """k - q up to 4/3: the pair densities' sphere leaves the box of the caller's
    grid, whose own representation of those components defines the result"""
    s = synth.small(method, nr=(16, 16, 16), tr=True, ecut=5.0, nbands=2, nocc=1)
    check(s, abi.TERMS_HF if method == "HF" else abi.TERMS_TC, prec, 12 if method == "HF" else 16)


def at_edge(n, fac):
    """cutoff for which n^3 is the smallest grid with periods longer than fac R"""
    return 0.5 * (0.985 * n * np.sqrt(3.0) * 2.0 * np.pi / 10.26 / fac) ** 2


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,user", [(15, 20), (15, 15), (27, 32), (45, 48)])
def test_work_grid_of_uneven_lines(n, user, prec):
    """n^3 is the smallest work grid; the next size is taken where n's lines split
    badly (15, in FP64 27 and 45)"""
    s = synth.small("TC", nr=(user, user, user), nk=1, ecut=at_edge(n, 6.0), nbands=2, nocc=1, seed=n)
    edge = {(15, 20): 16, (15, 15): 15, (27, 32): 30, (45, 48): 48}[n, user] if prec == "fp64" or n == 15 else n
    check(s, abi.TERMS_TC, prec, edge)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method", ["HF", "TC"])
@pytest.mark.parametrize("n,user", [(15, 16), (27, 30), (45, 48), (25, 27)])
def test_work_grid_next_to_the_callers(n, user, method, prec):
    """where the size that replaces a badly splitting one is the caller's own, the
    caller's grid stays; other sizes one step below the caller's are taken (when they
    save a tenth of the points)"""
    s = synth.small(method, nr=(user, user, user), nk=1, ecut=at_edge(n, 6.0 if method == "TC" else 4.0), nbands=1, nocc=1)
    stay = n == 15 or (prec == "fp64" and (n == 27 or (n == 45 and method == "TC")))
    with Context(s, prec) as ctx:
        assert ctx.work_grid() == ((user if stay else n),) * 3


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("method,F", [("TC", 1.2), ("BITC", 1.2), ("BITC", np.array([[1.3, 1.0], [1.0, 1.2]]))])
def test_work_grid_spin_channels(method, F, prec):
    """two spin channels, equal and unequal Jastrow channels, on a smaller grid"""
    s = synth.small(method, nr=(24, 24, 24), nk=2, ecut=3.5, nbands=2, nocc=1, nspin=2, F=F, seed=8)
    check(s, abi.TERMS_TC, prec, 16)


def refine(s, n):
    """the system on a finer n^3 grid, with the density of its orbitals there"""
    n0 = np.array(s.nr)
    w = np.stack([s.gindex % n0[0], (s.gindex // n0[0]) % n0[1], s.gindex // (n0[0] * n0[1])], 1)
    m = np.mod(np.where(w > n0 // 2, w - n0, w), n)
    s = dataclasses.replace(s, nr=(n, n, n), gindex=(m[:, 0] + n * (m[:, 1] + n * m[:, 2])).astype(np.int32))
    s.density = O.density(s)
    return s


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("term", ["hf2x", "tc2x", "tc3a1", "tc3b1", "tc3a2a4b2b5", "tc3a3b3b4b6"])
def test_work_grid_of_a_symmetry_reduced_run(term, prec):
    """silicon with rotations and the (1/4, 1/4, 1/4) translation, on a caller's grid
    fine enough for a smaller work grid (a multiple of 4 for TC / BITC, on which the
    translation is integral)"""
    from test_qe_symmetry import qe_system
    if term not in _qe:
        s = refine(qe_system("HF" if term == "hf2x" else "BITC"), 24)
        _qe[term] = s, O.apply(s, abi.TERM_NAMES[term])
    s, (r2, r3) = _qe[term]
    with Context(s, prec) as ctx:
        ctx.set_state()
        assert ctx.work_grid() == ((16,) * 3 if term == "hf2x" else (20,) * 3)
        g2, g3 = ctx.apply(abi.TERM_NAMES[term])
    ref, got = (r2, g2) if abi.TERM_NAMES[term] & abi.TERMS_H2 else (r3, g3)
    assert rel(got, ref) < TOL[prec]


_qe = {}


@pytest.mark.parametrize("amplitude,edge", [(3e-14, 16), (3e-13, 24)])
def test_density_at_the_threshold(amplitude, edge):
    """a component beyond the pair densities' sphere just below 1e-13 of the largest is
    dropped with the smaller grid, just above it the caller's grid is used; either
    way the results are the oracle's for that density"""
    s = synth.small("TC", nr=(24, 24, 24), nk=1, ecut=3.5, nbands=2, nocc=2, seed=4)
    wave = 2.0 * amplitude * s.density[0].real.mean() * np.cos(2 * np.pi * 10 * (np.arange(s.N) % 24) / 24.0)
    s.density = s.density + wave[None, :]
    check(s, abi.TERMS_TC, "fp64", edge)


def test_density_beyond_the_pair_sphere():
    """a density with a component outside the pair densities' sphere needs the
    caller's grid; the next state may go back to the smaller one"""
    s = synth.small("TC", nr=(32, 32, 32), nk=1, ecut=6.0, nbands=2, nocc=2, seed=4)
    plain = s.density.copy()
    z, y, x = np.meshgrid(*[np.arange(32) / 32.0] * 3, indexing="ij")
    wave = 0.05 * np.abs(plain).max() * np.cos(2 * np.pi * (13 * x + 2 * y - 11 * z)).ravel()
    with Context(s, "fp64") as ctx:
        small = ctx.work_grid()
        assert small[0] < 32
        for dens, grid in ((plain, small), (plain + wave[None, :], (32,) * 3), (plain, small)):
            s.density = dens
            r2, r3 = O.apply(s, abi.TERMS_TC)
            ctx.set_state()
            assert ctx.work_grid() == grid
            g2, g3 = ctx.apply(abi.TERMS_TC)
            assert rel(g2, r2) < TOL["fp64"]
            assert rel(g3, r3) < TOL["fp64"]
    s.density = plain


@pytest.mark.parametrize("nr,edge", [((18, 20, 16), None), ((16, 24, 18), None), ((30, 30, 30), 24)])
def test_pencils_of_the_pair_balls(nr, edge):
    """the table of needed pencils (several k-differences, unequal sides): the pruned
    transforms give what the full ones give, up to the rounding of FP64"""
    s = synth.small("TC", nr=nr, nk=2, ecut=4.0 if edge is None else 7.0, nbands=2, nocc=1, seed=2)
    out = []
    with Context(s, "fp64") as ctx:
        if edge:
            assert ctx.work_grid() == (edge,) * 3
        for prune in (1, 0):
            ctx.set_forms(prune=prune)
            ctx.set_state()
            out.append(ctx.apply(abi.TERMS_TC))
    assert rel(out[0][0], out[1][0]) < 1e-12
    assert rel(out[0][1], out[1][1]) < 1e-12


def test_refused_pseudopotential_and_grid_change():
    """a local potential that is refused (NaN) leaves none: the next state may change
    the work grid, and the terms of an earlier pseudopotential are gone"""
    s = synth.small("TC", nr=(32, 32, 32), nk=1, ecut=6.0, nbands=2, nocc=2, seed=4)
    good, bad = synth.pseudo(s), synth.pseudo(s)
    bad.vloc = np.where(np.arange(s.N) == 5, np.nan, bad.vloc)
    z, y, x = np.meshgrid(*[np.arange(32) / 32.0] * 3, indexing="ij")
    plain = s.density.copy()
    wave = 0.05 * np.abs(plain).max() * np.cos(2 * np.pi * (13 * x + 2 * y - 11 * z)).ravel()
    for first in (None, good):
        with Context(s, "fp64") as ctx:
            if first is not None:
                ctx.set_pseudo(first)
            with pytest.raises(TCError) as e:
                ctx.set_pseudo(bad)
            assert e.value.code == abi.TCG_ERR_NUMERIC
            with pytest.raises(TCError) as e:
                ctx.apply_h1(abi.TERM_PSEUDO)
            assert e.value.code == abi.TCG_ERR_STATE
            for dens in (plain + wave[None, :], plain):
                s.density = dens
                r2, _ = O.apply(s, abi.TERM_TC2X)
                ctx.set_state()
                assert rel(ctx.apply(abi.TERM_TC2X)[0], r2) < TOL["fp64"]
            ctx.set_pseudo(good)
            assert rel(ctx.apply_h1(abi.TERM_PSEUDO), O.apply_h1(s, abi.TERM_PSEUDO, good)) < TOL["fp64"]
    s.density = plain


@pytest.mark.parametrize("how", ["set_state", "set_forms"])
def test_failed_allocation_during_a_grid_change(how):
    """each allocation of a state that moves to another work grid fails in turn (on the
    host): there is no state afterwards, and the next one is right"""
    import ctypes
    from tc_b200._lib import lib
    arm = lib().tcg_debug_fail_alloc
    arm.argtypes, arm.restype = [ctypes.c_int32], None
    s = synth.small("TC", nr=(24, 24, 24), nk=1, ecut=3.5, nbands=2, nocc=2, seed=4)
    plain = s.density.copy()
    beyond = plain + 0.05 * np.abs(plain).max() * np.cos(2 * np.pi * 10 * (np.arange(s.N) % 24) / 24.0)[None, :]
    d0 = O.density(s)
    s.density = beyond
    r2, r3 = O.apply(s, abi.TERMS_TC)
    p2, p3 = O.apply(dataclasses.replace(s, density=plain), abi.TERMS_TC)
    failures = 0
    for nth in range(1, 200):
        s.density = plain
        with Context(s, "fp64") as ctx:
            ctx.set_state()
            if how == "set_state":
                s.density, want = beyond, (r2, r3)
            else:
                want = (p2, p3)
            arm(nth)
            try:
                if how == "set_state":
                    ctx.set_state()
                else:
                    ctx.set_forms(xy=1)                    # takes the state to the caller's grid
            except TCError as e:
                assert e.code == abi.TCG_ERR_NOMEM
            else:
                break
            finally:
                arm(0)
            failures += 1
            for call in (lambda: ctx.apply(abi.TERMS_TC), ctx.refresh_state, ctx.qp_finish):
                with pytest.raises(TCError) as e:
                    call()
                assert e.value.code == abi.TCG_ERR_STATE
            assert rel(ctx.density(), d0) < 1e-12
            assert rel(ctx.apply_h1(abi.TERM_KINETIC), O.apply_h1(s, abi.TERM_KINETIC)) < TOL["fp64"]
            ctx.set_state()
            g2, g3 = ctx.apply(abi.TERMS_TC)
            assert rel(g2, want[0]) < TOL["fp64"]
            assert rel(g3, want[1]) < TOL["fp64"]
    s.density = plain
    assert failures >= 8                                   # twiddles, maps, density, orbital grids, local potentials


def test_no_stage_survives_its_state():
    """the occupied-pair stage begun for a state is gone with it"""
    s = synth.small("TC", nr=(12, 12, 12), nk=1, ecut=2.5, nbands=2, nocc=2, seed=4)
    with Context(s, "fp64") as ctx:
        ctx.set_state()
        ctx.qp_partial(0, 1)
        ctx.density()
        with pytest.raises(TCError) as e:
            ctx.qp_finish()
        assert e.value.code == abi.TCG_ERR_STATE


@pytest.mark.parametrize("method", ["HF", "TC", "BITC"])
def test_density_from_the_work_grid(method):
    s = synth.small(method, nr=(32, 32, 32), nk=2, ecut=5.0, nbands=2, nocc=2, seed=6)
    d0 = O.density(s)
    with Context(s, "fp64") as ctx:
        d = ctx.density()
    assert rel(d, d0) < 1e-12


@pytest.mark.parametrize("npw,nbasis,nblock", [(40, 3, 9), (512, 8, 8), (1025, 5, 17), (3073, 1, 3), (5121, 2, 10)])
def test_expansion_edges(npw, nbasis, nblock):
    """block Gram-Schmidt at the edges of its register tiles and panels, with a
    vector that vanishes, against numpy (1e-10)"""
    import torch
    from tc_b200.context import davidson_expand
    rng = np.random.default_rng(npw)
    V0 = np.linalg.qr(rng.standard_normal((npw, nbasis)) + 1j * rng.standard_normal((npw, nbasis)))[0].T
    phi = rng.standard_normal((nblock, npw)) + 1j * rng.standard_normal((nblock, npw))
    H = rng.standard_normal((nblock, npw)) + 1j * rng.standard_normal((nblock, npw))
    kg2 = rng.uniform(0.1, 20.0, npw)
    eig = rng.standard_normal(nblock) + 0j
    if nblock > 2:
        phi[2], H[2], eig[2] = phi[1], H[1], eig[1]          # the same residual twice: dropped
    rows = [v for v in V0]
    for b in range(nblock):
        x = kg2 / (np.sum(kg2 * np.abs(phi[b]) ** 2) / np.sum(np.abs(phi[b]) ** 2))
        p = 27 + x * (18 + x * (12 + 8 * x))
        t = -(p / (p + 16 * x ** 4)) * (H[b] - eig[b] * phi[b])
        t /= np.linalg.norm(t)
        for v in rows:
            t = t - np.vdot(v, t) * v
        if np.linalg.norm(t) >= 1e-8:
            rows.append(t / np.linalg.norm(t))
    V = torch.zeros((nbasis + nblock, npw), dtype=torch.complex128, device="cuda")
    V[:nbasis] = torch.from_numpy(np.ascontiguousarray(V0)).cuda()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    n = davidson_expand(V, nbasis, dev(phi), [dev(H)], dev(kg2), eig)
    assert n == len(rows)
    assert np.abs(V[:n].cpu().numpy() - np.array(rows)).max() < 1e-10


@pytest.mark.parametrize("scale", [0.0, 1e-170, 1e-110, 1e110, 1e150])
@pytest.mark.parametrize("n", [3, 17, 96])
@pytest.mark.parametrize("real", [False, True])
def test_subspace_eigen_of_extreme_norm(n, scale, real):
    """matrices whose squared elements under- or overflow; eigenvalues and residual in
    units of the scale, tolerance as in test_subspace_eigen"""
    import torch
    from tc_b200.context import subspace_ritz
    rng = np.random.default_rng(n)
    H = (rng.standard_normal((n, n)) + (0j if real else 1j) * rng.standard_normal((n, n))) * (scale > 0)
    V = np.eye(n, n + 5, dtype=complex)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    w, _, Vo, _ = subspace_ritz(dev(V), [dev(scale * H.T @ V), None, None], n)
    X = Vo.cpu().numpy()[:, :n].T
    w = w / scale if scale else w
    assert np.abs(np.linalg.norm(X, axis=0) - 1.0).max() <= 1e-12
    assert np.abs(H @ X - X * w).max() <= 50 * n * 2.2e-16 * np.linalg.norm(H)


@pytest.mark.parametrize("kind", ["general", "hermitian", "degenerate", "triangular"])
@pytest.mark.parametrize("n", [1, 2, 3, 17, 32, 33, 64, 96, 112, 113])
def test_subspace_eigen(n, kind):
    """the one-CTA eigensolve (up to order 112) and the library's beyond: with unit
    vectors as the basis the Ritz vectors are the eigenvectors themselves.
    |H X - X D| is the backward error of a QR iteration, some n eps |H|."""
    import torch
    from tc_b200.context import subspace_ritz
    rng = np.random.default_rng(n)
    H = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "hermitian":
        H = H + H.conj().T
    elif kind == "degenerate":
        Q = np.linalg.qr(H)[0]
        H = (Q * np.repeat(np.arange(n), 3)[:n]) @ Q.conj().T
    elif kind == "triangular":
        H = np.triu(H) + 3.0 * np.diag(np.arange(n))
    V = np.eye(n, n + 5, dtype=complex)
    HV = H.T @ V                                          # row j: H V_j
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    w, e, Vo, _ = subspace_ritz(dev(V), [dev(HV), None, None], n)
    X = Vo.cpu().numpy()[:, :n].T
    nrm = np.linalg.norm(H)
    assert np.all(np.diff(w.real) >= 0)
    assert np.abs(np.linalg.norm(X, axis=0) - 1.0).max() <= 1e-12
    assert np.abs(H @ X - X * w).max() <= 50 * n * 2.2e-16 * nrm

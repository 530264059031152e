"""Sums over the occupied orbitals in the mixed path: their rounding must not
grow with the number of orbitals.

A state of n copies of one orbital with filling f / n (n a power of two) sums n
equal terms, each the single orbital's divided by n without rounding.  FP32 sums
cover at most 8 sources, the rest is added in FP64: with n = 8 and with n = 128
every group then rounds alike, and the FP64 sum of equal groups is exact.  So the two states give the same H2 up to the rounding of FP64 (1e-12) and
the same H3 up to that of an FP32 copy of a sum whose value lies on the border of
two FP32 numbers (1.2e-7 at one of 1728 points or more: below 1e-8).  An FP32 sum
over more sources rounds the two differently, by some 1e-7 at every point."""
import numpy as np
import pytest

from tc_b200 import abi, synth
from tc_b200.context import Context

pytestmark = pytest.mark.gpu


def copies(s, n, f):
    """the state with n copies of the occupied orbital of s, filling f / n each"""
    s.nbands = np.full(s.nspin, n, dtype=np.int32)
    s.nocc = np.full((s.nspin, s.nk_irr), n, dtype=np.int32)
    s.filling = np.full(s.nspin * s.nk_irr * n, f / n)
    rep = lambda x: np.concatenate([np.tile(o, n) for o in np.split(x, np.cumsum(np.tile(s.npw, s.nspin))[:-1])])
    s.phik = rep(s.phik)
    if s.phik_left is not None:
        s.phik_left = rep(s.phik_left)
    return s


def run(method, nr, n, f, ntarget=2, terms=None, ecut=3.0, **kw):
    s = synth.small(method, nr=nr, nk=1, ecut=ecut, nbands=1, nocc=1, seed=3, **kw)
    psi = synth.small(method, nr=nr, nk=1, ecut=ecut, nbands=ntarget, nocc=1, seed=5, **kw).psi if ntarget <= 8 else \
        np.random.default_rng(5).standard_normal(2 * int(s.npw.sum()) * s.nspin * ntarget).view(np.complex128)
    copies(s, n, f)
    s.nb_apply = np.full((s.nspin, s.nk_irr), ntarget, dtype=np.int32)
    s.psi = psi
    if terms is None:
        terms = abi.TERMS_HF if method == "HF" else abi.TERMS_TC
    with Context(s, "mixed") as ctx:
        ctx.set_state()
        return ctx.apply(terms)


def rel2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


UNEQUAL = dict(nspin=2, F=np.array([[1.3, 1.0], [1.0, 1.2]]))


@pytest.mark.parametrize("method,nr,kw", [
    ("HF", (12, 12, 12), {}), ("HF", (24, 24, 24), {}), ("HF", (14, 14, 14), dict(ecut=6.0)),
    ("TC", (12, 12, 12), {}), ("TC", (20, 20, 20), {}), ("TC", (14, 15, 12), {}), ("TC", (12, 12, 12), UNEQUAL),
    ("TC", (14, 15, 12), UNEQUAL), ("BITC", (15, 15, 15), {}), ("BITC", (14, 15, 12), UNEQUAL)])
def test_rounding_of_many_sources(method, nr, kw):
    a2, a3 = run(method, nr, 8, 2.0, **kw)
    b2, b3 = run(method, nr, 128, 2.0, **kw)
    assert rel2(b2, a2) <= 1e-12
    if method != "HF":
        assert rel2(b3, a3) <= 1e-8


def test_rounding_of_many_sources_and_targets():
    """as many targets as leave the on-chip hf2x one CTA per target"""
    a2, _ = run("HF", (12, 12, 12), 8, 2.0, ntarget=1300)
    b2, _ = run("HF", (12, 12, 12), 128, 2.0, ntarget=1300)
    assert rel2(b2, a2) <= 1e-12


@pytest.mark.parametrize("method,nr", [("HF", (12, 12, 12)), ("HF", (25, 25, 25)), ("TC", (12, 12, 12)), ("TC", (14, 15, 12))])
def test_fillings_are_not_rounded(method, nr):
    """fillings of 0.3 (no FP32 number: 4e-8 off) and 0.25 give H2 in the ratio 6 / 5.
    Rounding of single points averages out over 1728 points and more to below 1e-9."""
    t = abi.TERM_HF2X if method == "HF" else abi.TERM_TC2X
    a, _ = run(method, nr, 2, 0.6, terms=t)
    b, _ = run(method, nr, 2, 0.5, terms=t)
    assert abs(np.vdot(b, a).real / np.vdot(b, b).real / 1.2 - 1.0) <= 5e-9

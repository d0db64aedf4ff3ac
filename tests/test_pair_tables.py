"""The FP64 pair sweeps from tabulated functions of r^2 (pair64.cu): the table
over its whole range and past its ends, and the sweeps' lane splits, queues of
put-aside pairs and energy splits at the sizes where they change, against the
oracle's written-out expressions.

Tolerances: a table value is off by one rounding and 2^-54; force and energy of
a pair by about five roundings, the oracle's by as many: 1e-14 of a single
pair's force.  Sums over an atom's rows: the parity tests' 1e-10, tightened to
1e-12 of the largest force (up to 10^3 terms of 1e-16)."""
import dataclasses

import numpy as np
import pytest

import oracle
from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64
from tests import systems


def _two_ions():
    spec = S.RunSpec(molecules=[("Cl-", 2)], box=(40.0, 40.0, 40.0), dt_fs=2.0, nfreq=1,
                     rcut=12.0, rshort=12.0, alpha=0.28 * 12.0, fexp=1.0, ichnb=10, trtemp=300.0)
    return S.System(spec)


@pytest.mark.gpu
def test_pair_table_range():
    """Two ions from 0.3 A (below the table: written out) to 12 A: force and
    energies of LOCALF; bin edges among the distances."""
    from mdynamix_gb300.mdx import ForcePath
    s = _two_ions()
    g, o = ForcePath(s, precision=MDX_FP64), oracle.Oracle(s)
    z = np.zeros(2)
    r = list(np.exp(np.linspace(np.log(0.3), np.log(11.99), 150)))
    r += [np.sqrt(v) for v in (0.25, np.nextafter(0.25, 0), 1.0, 1.0078125, 16.0, 127.5)]
    for d in r:
        st = (np.array([-0.5 * d, 0.5 * d]), z, z, z, z, z)
        for p in (g, o):
            p.set_state(*st)
            p.chcnb()
            p.getcom()
        a, b = g.fforces(), o.fforces()
        fa, fb = g.forces(1), o.forces(1)
        # the force's parts, which nearly cancel near 11 A: the screened Coulomb
        # term is at least TOTPI alpha exp(-(alpha r)^2) QIJ / r, the LJ terms
        # A6 and B12 apart
        i = s.inbt[0] - 1
        parts = (s.coulf * 1.128379169 * s.alphad * np.exp(-(s.alphad * d) ** 2) / d
                 + abs(6 * s.a6lj[i, i]) / d ** 7 + abs(12 * s.b12lj[i, i]) / d ** 13)
        assert np.abs(fa - fb).max() <= 2e-14 * parts, d
        assert abs(a.pels2 - b.pels2) <= 1e-14 * abs(b.pels2), d


@pytest.mark.gpu
@pytest.mark.parametrize("nw,kind", [(8, "water"), (203, "water"), (833, "water"), (1650, "water"),
                                     (300, "organics"), (1640, "organics"), (300, "skin"),
                                     (833, "ee")])
def test_pair_sweeps_match_oracle(nw, kind):
    """Lane splits of the short rows (32, 16, 8 lanes at about 2,400 and 4,900
    atoms), queues that fill and that end part full (organics: own-molecule,
    1-4 and many LJ pairs; ee: pairs shifted by MDEE), rows of no entries, the
    skin's cutoff; energies by type pair from the force calls."""
    from mdynamix_gb300.mdx import ForcePath
    spec = systems.spcfw(n=nw, ions=2, rcut=7.0 if nw < 100 else 8.0)
    if nw < 100:
        spec = dataclasses.replace(spec, box=(30.0, 30.0, 30.0))
    if kind == "organics":
        spec = dataclasses.replace(systems.organics(nw), molecules=[
            ("H2O", nw), ("CH3OH", 3 + nw // 200), ("C2H5OH", 2 + nw // 300)])
    if kind == "skin":
        spec = dataclasses.replace(systems.spcfw(n=512, rcut=9.0), rskin=1.5)
    if kind == "ee":
        spec = dataclasses.replace(S.solvation_job("C2H5OH", nw), rcut=8.0)
    s, st = systems.build(spec)
    g, o = ForcePath(s, precision=MDX_FP64), oracle.Oracle(s, threads=4)
    for p in (g, o):
        if kind == "ee":
            p.set_lambda(0.5)
        p.set_state(*st)
        p.chcnb()
        p.getcom()
    for routine, which in (("fforces", 1), ("slforces", 2), ("allforce", 3)):
        a, b = getattr(g, routine)(), getattr(o, routine)()
        fa, fb = g.forces(which), o.forces(which)
        assert np.abs(fa - fb).max() <= 1e-12 * np.abs(fb).max(), routine
        names = {"fforces": ("pels2", "pe2", "vir2"), "slforces": ("pels1", "pe1", "vir1"),
                 "allforce": ("pels1", "pe1", "pels2", "pe2")}[routine]
        for n in names:
            assert abs(getattr(a, n) - getattr(b, n)) <= 1e-10 * max(abs(getattr(b, n)), 1e-9), n
        for n in ("pote1", "potl1", "pes141", "psr141"):
            x, y = np.array(getattr(a, n)), np.array(getattr(b, n))
            assert np.abs(x - y).max() <= 1e-10 * max(np.abs(y).max(), 1e-9), (routine, n)


@pytest.mark.gpu
@pytest.mark.parametrize("nw,kind", [(8, "water"), (203, "water"), (300, "organics"), (300, "ee"),
                                     (1650, "water")])
def test_mixed_energies_by_type_pair(nw, kind):
    """POTE1, POTL1, PES141, PSR141 of the mixed path's force calls (a slot's
    sums kept per lane) against the FP64 path: rows whose partners change type
    (ions, organics), own-molecule and 1-4 pairs, the MDEE sweeps.  A term is
    good to a few 1e-6 (FP32 from 32-bit coordinates); the sums to 1e-4 of the
    largest, the mixed path's energy bound."""
    from mdynamix_gb300.abi import MDX_MIXED
    from mdynamix_gb300.mdx import ForcePath
    spec = systems.spcfw(n=nw, ions=2, rcut=7.0 if nw < 100 else 8.0)
    if nw < 100:
        spec = dataclasses.replace(spec, box=(30.0, 30.0, 30.0))
    if kind == "organics":
        spec = systems.organics(nw)
    if kind == "ee":
        spec = dataclasses.replace(S.solvation_job("C2H5OH", nw), rcut=8.0)
    s, st = systems.build(spec)
    out = []
    for prec in (MDX_FP64, MDX_MIXED):
        g = ForcePath(s, precision=prec)
        if kind == "ee":
            g.set_lambda(0.5)
        g.set_state(*st)
        g.chcnb()
        g.getcom()
        out.append(g.allforce())
        g.close()
    a, b = out
    for n in ("pote1", "potl1", "pes141", "psr141"):
        x, y = np.array(getattr(a, n)), np.array(getattr(b, n))
        assert np.abs(x - y).max() <= 1e-4 * max(np.abs(x).max(), 1e-9), n


@pytest.mark.gpu
@pytest.mark.parametrize("box", [(40.0, 40.0, 40.0), (31.0, 45.0, 38.0), (200.0, 60.0, 90.0)])
def test_fixed_point_pairs(box):
    """Two ions across the faces of the cell, from 0.3 A (written out; large LJ
    forces) through the starts and ends of the sweeps' ranges to 12 A, cut at
    5 A between LOCALF and FORCES.  A pair's force: 2^-53 of the Coulomb force
    at its sweep's first r^2 (2 and 16 A^2: three roundings of a quarter of
    that) beside the 2e-14 of its parts; energies alike."""
    from mdynamix_gb300.mdx import ForcePath
    # no k-vectors: G is the pair force alone
    spec = dataclasses.replace(_two_ions().spec, box=box, rshort=5.0, fexp=1e-4)
    s = S.System(spec)
    g, o = ForcePath(s, precision=MDX_FP64), oracle.Oracle(s)
    i = s.inbt[0] - 1
    rng = np.random.default_rng(3)
    r = list(np.exp(np.linspace(np.log(0.3), np.log(11.99), 120)))
    r += [np.sqrt(v) for v in (1.9999999, 2.0, 2.015625, 15.9999, 16.0, 24.999, 25.001, 63.99)]
    for d in r:
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        c = 0.5 * np.array(box) * rng.choice([-1.0, 1.0], 3) + rng.normal(size=3)
        xy = np.stack([c - 0.5 * d * u, c + 0.5 * d * u], 1)
        st = tuple(xy) + (np.zeros(2),) * 3
        for p in (g, o):
            p.set_state(*st)
            p.chcnb()
            p.getcom()
        for routine, which, r0, names in (("fforces", 1, 2.0, ("pels2", "virfx")),
                                          ("slforces", 2, 16.0, ("pels1",))):
            a, b = getattr(g, routine)(), getattr(o, routine)()
            fa, fb = g.forces(which), o.forces(which)
            coul = s.coulf * 1.128379169 * s.alphad * np.exp(-(s.alphad * d) ** 2) / d
            parts = (coul + abs(6 * s.a6lj[i, i]) / d ** 7 + abs(12 * s.b12lj[i, i]) / d ** 13)
            start = s.coulf / r0
            tol = 2e-14 * parts + 2.0 ** -53 * start
            assert np.abs(fa - fb).max() <= tol, (routine, d)
            assert abs(getattr(a, names[0]) - getattr(b, names[0])) <= (
                1e-14 * abs(getattr(b, names[0])) + 2.0 ** -53 * start * np.sqrt(r0)), (routine, d)

"""Bonded terms, a thread a term (FFORCES without statistics): molecule counts at
the edges of its blocks, straight angles (CH3CN as built and bent).  FP64 against
the oracle: a term's force takes some 30 roundings and the sine of a nearly
straight angle is conditioned like the angle itself: 1e-11 of the largest
force.  Mixed (bent molecules) against FFORCES with statistics, whose threads
take a molecule: the same FP32 terms but for the contraction of their some 30
operations, 30 x 2^-24 of the largest force."""
import numpy as np
import pytest

import oracle
from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129])
@pytest.mark.parametrize("jitter,prec", [(0.0, MDX_FP64), (0.03, MDX_FP64), (0.03, MDX_MIXED)])
def test_terms(n, jitter, prec):
    from mdynamix_gb300.mdx import ForcePath
    box = 14.0 + 9.0 * n ** (1 / 3)
    first = "CH3CN" if prec == MDX_FP64 else "CH3OH"
    spec = S.RunSpec(molecules=[(first, n), ("SPC-FW", n), ("C2H5OH", 2)], box=(box,) * 3,
                     dt_fs=1.0, nfreq=4, rcut=6.5, rshort=4.0, alpha=2.0, fexp=1.0, ichnb=10,
                     trtemp=300.0)
    s = S.System(spec)
    st = S.make_configuration(s, seed=6, jitter=jitter)
    g = ForcePath(s, precision=prec)
    o = oracle.Oracle(s) if prec == MDX_FP64 else None
    for p in (g, o) if o else (g,):
        p.set_state(*st)
        p.chcnb()
        p.getcom()
        p.fforces(False)
    a = g.forces(1)
    if o:
        b = o.forces(1)
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
    else:
        g.fforces(True)
        b = g.forces(1)
        assert np.abs(a - b).max() <= 30 * 2.0 ** -24 * np.abs(b).max()
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
def test_bond_of_no_length(prec):
    """A frozen molecule with two sites in one place: the bond's energy is finite and
    no force comes of it.  Energy: FP64 as the terms above, mixed 30 x 2^-24."""
    from mdynamix_gb300.mdx import ForcePath
    spec = S.RunSpec(molecules=[("SPC_E", 3), ("Na+", 2)], box=(20.0,) * 3, dt_fs=1.0, nfreq=4,
                     rcut=6.5, rshort=4.0, alpha=2.0, fexp=1.0, ichnb=10, trtemp=300.0,
                     lmove=[0, 1])
    s = S.System(spec)
    st = [a.copy() for a in S.make_configuration(s, seed=6, jitter=0.0)]
    for a in st[:3]:
        a[4] = a[3]  # the second water's first hydrogen on its oxygen
    g, o = ForcePath(s, precision=prec), oracle.Oracle(s)
    for p in (g, o):
        p.set_state(*st)
        p.chcnb()
        p.getcom()
    a, b = g.fforces(False), o.fforces(False)
    assert b.pint > 0.0 and np.isfinite(g.forces(1)).all()
    assert abs(a.pint - b.pint) <= (1e-11 if prec == MDX_FP64 else 30 * 2.0 ** -24) * b.pint
    g.close()

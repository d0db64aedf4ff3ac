"""Per-molecule passes with several lanes per molecule (kick + drift + GETCOM,
SCALING's molecular correction, SHEJK): molecules of 1, 3-4, 5-16, 17-32 and
more atoms in one system, on both paths.  Against the oracle's loops: the FP64
path to the parity tests' 1e-9 A after a few steps (sums of up to 118 terms in
another order: 1e-14), the mixed path to 1e-5 A."""
import dataclasses

import numpy as np
import pytest

import oracle
from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED


def _sizes():
    """One molecule name for each lane count (1, 4, 8, 16, 32)."""
    db = S.load_moldb()
    pick = {}
    for name, m in sorted(db.items()):
        n = len(m["sites"])
        g = 1 if n == 1 else 4 if n <= 4 else 8 if n <= 16 else 16 if n <= 32 else 32
        if n != 2 and (g not in pick or n < len(db[pick[g]]["sites"])):
            pick[g] = name
    return pick


def _start(npt):
    names = _sizes()
    mols = [(names[g], 2 if g > 8 else 5) for g in sorted(names)]
    spec = S.RunSpec(molecules=mols, box=(60.0, 60.0, 60.0), dt_fs=0.5, nfreq=1 if npt else 4,
                     rcut=9.0, rshort=5.0, alpha=2.5, fexp=4.0, ichnb=10, nvt=(300.0, 30.0),
                     npt=(1.0, 1000.0) if npt else None, anisotropic=npt, trtemp=300.0,
                     shake=npt, shake_hbonds=npt, toler=1e-5)
    s = S.System(spec)
    return s, S.make_configuration(s, seed=5, jitter=0.02)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
@pytest.mark.parametrize("npt", [False, True])
def test_lanes_per_molecule(npt, prec):
    from mdynamix_gb300.mdx import ForcePath
    s, st = _start(npt)
    assert set(s.nsits) and max(s.nsits) > 32
    g, o = ForcePath(s, precision=prec), oracle.Oracle(s)
    for p in (g, o):
        p.set_state(*st)
        (p.sultan if npt else p.double)(3)
    (x, y, z, *v), _ = g.get_state()
    (ox, oy, oz, *ov), _ = o.get_state()
    d = max(np.abs(x - ox).max(), np.abs(y - oy).max(), np.abs(z - oz).max())
    assert d < (1e-9 if prec == MDX_FP64 else 1e-5), d
    dv = max(np.abs(a - b).max() for a, b in zip(v, ov)) / max(np.abs(b).max() for b in ov)
    assert dv < (1e-9 if prec == MDX_FP64 else 1e-4), dv

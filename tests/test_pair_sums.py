"""Energies and virials of the FP64 pair sweeps, whose terms nearly cancel, against
sums in long double over every pair.

Tolerance: an FP64 sum of terms of some five roundings each is off by about 2^-53 of
the root of the sum of the terms' squares, and by a few times that for the additions
of its partial sums; 32 times is held."""
import copy

import numpy as np
import pytest

from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64

A = [np.longdouble(v) for v in (0.254829592, -0.284496736, 1.421413741, -1.453152027,
                                1.061405429)]


def _exact(s, pos, box, rcut, rshort):
    """(terms' sum, root of their squares' sum) of the diagonal virial and the Coulomb
    energy, short rows then long."""
    n, ld = len(pos), np.longdouble
    i, j = np.triu_indices(n, 1)
    d = pos[i] - pos[j]
    d -= box * np.round(d / box)
    keep = (d ** 2).sum(1) <= rcut * rcut
    i, j = i[keep], j[keep]
    d = pos[i].astype(ld) - pos[j].astype(ld)
    d -= ld(box) * np.round((d / ld(box)).astype(float))
    rr = (d ** 2).sum(1)
    r, al = np.sqrt(rr), ld(s.alphad)
    t, e = 1 / (1 + ld(0.3275911) * al * r), np.exp(-(al * r) ** 2)
    erfc = ((((A[4] * t + A[3]) * t + A[2]) * t + A[1]) * t + A[0]) * t * e
    e1 = ld(s.coulf) * s.q[i].astype(ld) * s.q[j].astype(ld) / r
    k = s.inbt[s.itype - 1] - 1  # one site a type
    a6, b12 = s.a6lj[k[i], k[j]].astype(ld), s.b12lj[k[i], k[j]].astype(ld)
    f = e1 * (ld(1.128379169) * al * e + erfc / r) / r + (6 * a6 + 12 * b12 / rr ** 3) / rr ** 4
    out = []
    for rows in (rr <= rshort ** 2, rr > rshort ** 2):
        terms = [f[rows] * d[rows, a] ** 2 for a in range(3)] + [(e1 * erfc)[rows]]
        out.append([(v.sum(), np.sqrt((v ** 2).sum())) for v in terms])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("charge", [1.0, 0.77])
@pytest.mark.parametrize("rshort", [3.5, 4.5])
def test_energy_and_virial_sums(rshort, charge):
    from mdynamix_gb300.mdx import ForcePath
    n, box, rcut = 1500, 31.0, 12.0
    s = copy.copy(S.System(S.RunSpec(
        molecules=[("Na+", n // 2), ("Cl-", n // 2)], box=(box,) * 3, dt_fs=2.0, nfreq=1,
        rcut=rcut, rshort=rshort, alpha=2.8, fexp=1e-5, ichnb=10, trtemp=300.0)))  # no k-vectors
    s.q, s.site_charge = np.asarray(s.q) * charge, np.asarray(s.site_charge) * charge
    rng = np.random.default_rng(1)
    cell = rng.permutation(12 ** 3)[:n]
    a = box / 12
    pos = (np.stack([cell // 144, (cell // 12) % 12, cell % 12], 1) + 0.5) * a - box / 2
    pos += rng.uniform(-0.12, 0.12, (n, 3)) * a
    short, long_ = _exact(s, pos, box, rcut, rshort)
    g = ForcePath(s, precision=MDX_FP64)
    g.set_state(*[np.ascontiguousarray(c) for c in pos.T], *[np.zeros(n)] * 3)
    g.chcnb()
    for sc, want, names in ((g.fforces(), short, ("virfx", "virfy", "virfz", "pels2")),
                            (g.slforces(), long_, ("virx", "viry", "virz", "pels1"))):
        for name, (total, scale) in zip(names, want):
            err = abs(np.longdouble(getattr(sc, name)) - total)
            assert err <= 32 * 2.0 ** -53 * scale, (name, float(err / (2.0 ** -53 * scale)))
    g.close()

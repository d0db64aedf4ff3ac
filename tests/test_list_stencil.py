"""CHCNB's stencil cut to the list sphere: the lists of both paths against the
oracle's, entry for entry, in boxes of 4 (scanned whole), 5, 6 and more list
cells an axis, atoms up to 3 A outside the box, and with 1-4 pairs and
exclusions.  Whole numbers: no tolerance."""
import numpy as np
import pytest

import oracle
from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
@pytest.mark.parametrize("box", [(17.6, 21.1, 31.0), (14.2, 35.3, 17.4), (24.6, 17.5, 14.0),
                                 (45.0, 18.0, 52.0)])
@pytest.mark.parametrize("rshort", [5.0, 7.5])
def test_lists_equal_oracle(box, rshort, prec):
    from mdynamix_gb300.mdx import ForcePath
    n = int(0.04 * np.prod(box)) // 2
    spec = S.RunSpec(molecules=[("C2H5OH", 4), ("Na+", n), ("Cl-", n)], box=box, dt_fs=1.0,
                     nfreq=4, rcut=7.0, rshort=rshort, alpha=2.0, fexp=4.0, ichnb=10,
                     trtemp=300.0)
    s = S.System(spec)
    st = list(S.make_configuration(s, seed=2, jitter=0.0))
    rng = np.random.default_rng(8)
    first = 4 * s.nsits[0]
    for a in range(3):  # the ions anywhere, some outside
        st[a][first:] = rng.uniform(-0.5 * box[a] - 3.0, 0.5 * box[a] + 3.0, 2 * n)
    caps = dict(cap_short=400, cap_long=600)
    g, o = ForcePath(s, precision=prec, **caps), oracle.Oracle(s)
    for p in (g, o):
        p.set_state(*st)
    assert g.chcnb() == o.chcnb()
    for a, b in zip(g.lists(), o.lists()):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
@pytest.mark.parametrize("far", [40.0, 1e5, 1e9, 3e12, float("inf"), float("nan")])
def test_far_positions(far, prec):
    """Atoms many boxes away, at infinity or nowhere: the other atoms' lists as the
    oracle's, which compares every pair (the mixed path's own are wrapped into the
    box); and RCUT below RSHORT."""
    from mdynamix_gb300.mdx import ForcePath
    for rcut in (7.0, 4.0):
        spec = S.RunSpec(molecules=[("Na+", 60), ("Cl-", 60)], box=(17.6, 21.1, 31.0), dt_fs=1.0,
                         nfreq=4, rcut=rcut, rshort=5.0, alpha=2.0, fexp=4.0, ichnb=10,
                         trtemp=300.0)
        s = S.System(spec)
        rng = np.random.default_rng(5)
        st = [rng.uniform(-0.5 * b, 0.5 * b, 120) for b in spec.box] + [np.zeros(120)] * 3
        for a in range(3):
            st[a][40 + a] = far
            st[a][90] = -far
        g, o = ForcePath(s, precision=prec), oracle.Oracle(s)
        for p in (g, o):
            p.set_state(*st)
            p.chcnb_counts = p.chcnb()
        if prec == MDX_MIXED and not far < 1e10:
            continue  # no place in 32-bit coordinates: the build only has to end
        for (x1, x2), (y1, y2) in zip(g.lists(), o.lists()):
            kx, ky = (~(np.isin(np.abs(u), [41, 42, 43, 91]) | np.isin(np.abs(v), [41, 42, 43, 91]))
                      for u, v in ((x1, x2), (y1, y2)))
            assert np.array_equal(x1[kx], y1[ky]) and np.array_equal(x2[kx], y2[ky])
        g.close()

"""The FP64 path at the sizes where its kernels change for large systems: the long
sweep's tables in shared memory (9,728 atoms and more) and one thread a molecule in
the kick and drift, with its clearing of the short sweep's sums (19,456 molecules
and more).  20,000 waters against the oracle, to the tolerances of the sweeps' and
the parity tests: forces 1e-12 of the largest, sums 1e-10, positions 1e-9 A."""
import numpy as np
import pytest

import oracle
from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64

pytestmark = pytest.mark.gpu


def test_forces_and_steps():
    from mdynamix_gb300.mdx import ForcePath
    s = S.System(S.RunSpec(molecules=[("SPC-FW", 20000)], density=1.0, dt_fs=2.0, nfreq=4,
                           rcut=8.0, rshort=5.0, alpha=2.4, fexp=2.0, ichnb=10,
                           nvt=(300.0, 30.0), trtemp=300.0))
    st = S.make_configuration(s, seed=9, jitter=0.05)
    g, o = ForcePath(s, precision=MDX_FP64), oracle.Oracle(s, threads=16)
    for p in (g, o):
        p.set_state(*st)
        p.getcom()
        p.counts_here = p.chcnb()
    assert g.counts_here == o.counts_here
    for routine, which, names in (
            ("fforces", 1, ("pels2", "pe2", "vir2", "pint")),
            ("slforces", 2, ("pels1", "pe1", "vir1", "virx", "wirs")),
            ("allforce", 3, ("pels1", "pels2", "pote1", "potl1"))):
        a, b = getattr(g, routine)(), getattr(o, routine)()
        fa, fb = g.forces(which), o.forces(which)
        assert np.abs(fa - fb).max() <= 1e-12 * np.abs(fb).max(), routine
        for n in names:
            x, y = np.atleast_1d(getattr(a, n)), np.atleast_1d(getattr(b, n))
            assert np.abs(np.array(x) - np.array(y)).max() <= 1e-10 * np.abs(y).max(), n
    for p in (g, o):
        p.set_state(*st)
        p.records = p.double(2)
    (x, y, z, *_), _ = g.get_state()
    (ox, oy, oz, *_), _ = o.get_state()
    assert max(np.abs(x - ox).max(), np.abs(y - oy).max(), np.abs(z - oz).max()) < 1e-9
    for n in ("pels1", "pe2", "pels2", "tke"):
        a, b = getattr(g.records[-1], n), getattr(o.records[-1], n)
        assert abs(a - b) <= 1e-10 * abs(b), n
    g.close()

"""The end of a DOUBLE step forms SLFORCES and FFORCES together (one clearing of
their sums, the pair sweeps' and k-vectors' sums folded by the kernels that form
them): its record against the two force calls on the final state.  FP64: the
same terms in another order, 1e-11.  Mixed: FP32 partial sums of up to 64 terms,
64 x 2^-24 of the terms' magnitudes, which for the short Coulomb energy of a
random water box add up to 450 times the energy: 2e-3."""
import numpy as np
import pytest

from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
@pytest.mark.parametrize("mols", [[("SPC-FW", 203)], [("C2H5OH", 1), ("SPC-FW", 120)]])
@pytest.mark.parametrize("averaging", [False, True])
def test_record_equals_force_calls(mols, prec, averaging):
    from mdynamix_gb300.mdx import ForcePath
    spec = S.RunSpec(molecules=mols, density=1.0, dt_fs=1.0, nfreq=4, rcut=7.0, rshort=4.5,
                     alpha=2.5, fexp=8.0, ichnb=10, nvt=(300.0, 30.0), trtemp=300.0)
    s = S.System(spec)
    g = ForcePath(s, precision=prec)
    g.set_state(*S.make_configuration(s, seed=4, jitter=0.03))
    if averaging:
        g.set_averaging(True)
    r = g.double(3)[-1]
    one = {"slow": g.slforces(), "fast": g.fforces(1)}
    tol = 1e-11 if prec == MDX_FP64 else 2e-3
    for call, names in (("slow", ("pe1", "pels1", "spe")), ("fast", ("pe2", "pels2", "pint"))):
        for n in names:
            a, b = getattr(r, n), getattr(one[call], n)
            assert abs(a - b) <= tol * abs(b), (n, a, b)
    g.close()

"""Set-up of the FP64 pair sweeps (their units and tables, pair64.cu) follows the
topology and the parameters, whatever the order of the calls.  Integer sums do
not depend on an order, so contexts that run the same sweeps in the same units
agree to the last bit: no tolerance."""
import copy
import ctypes as C
import dataclasses

import numpy as np
import pytest

from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, pack

pytestmark = pytest.mark.gpu


def _ions(n, box, fexp=1e-4):
    """Ions, LOCALF to 5 A; fexp 1e-4: no k-vectors."""
    return S.System(S.RunSpec(molecules=[("Na+", n), ("Cl-", n)], box=(box,) * 3, dt_fs=2.0,
                              nfreq=1, rcut=12.0, rshort=5.0, alpha=3.4, fexp=fexp, ichnb=10,
                              trtemp=300.0))


def _scaled(s, f):
    t = copy.deepcopy(s)
    t.q, t.site_charge = np.asarray(s.q) * f, np.asarray(s.site_charge) * f
    return t


def _evaluate(g, st):
    g.set_state(*st)
    g.chcnb()
    g.getcom()
    out = []
    for call, which, name in ((g.fforces, 1, "pels2"), (g.slforces, 2, "pels1")):
        sc = call()
        out.append((getattr(sc, name), g.forces(which)))
    return out


def _same(a, b):
    return all(x[0] == y[0] and np.array_equal(x[1], y[1]) for x, y in zip(a, b))


@pytest.mark.parametrize("scale", [1e-3, 0.125, 2.0])
@pytest.mark.parametrize("d", [3.0, 4.4, 7.7, 11.0])
def test_topology_again_with_other_charges(scale, d):
    """One pair of ions in either sweep, the charges of a second topology against
    a context that never had others."""
    from mdynamix_gb300.mdx import ForcePath
    s = _ions(1, 40.0)
    t = _scaled(s, scale)
    z = np.zeros(2)
    st = (np.array([-0.5 * d, 0.5 * d]), z, z, z, z, z)
    fresh, again = ForcePath(t, precision=MDX_FP64), ForcePath(s, precision=MDX_FP64)
    _evaluate(again, st)
    again._check(again.L.mdx_upload_topology(again.h, C.byref(pack(t, MDX_FP64).topo)))
    assert _same(_evaluate(fresh, st), _evaluate(again, st))
    fresh.close()
    again.close()


def test_parameters_before_topology():
    from mdynamix_gb300.mdx import ForcePath
    s = _ions(150, 30.0, fexp=4.0)
    st = S.make_configuration(s, seed=4, jitter=0.05)
    g, p = ForcePath(s, precision=MDX_FP64), ForcePath.__new__(ForcePath)
    a = _evaluate(g, st)
    assert _same(a, _evaluate(g, st))
    # the same context made by hand, parameters first
    p.L, p.system, p.n, p.packed = g.L, s, g.n, pack(s, MDX_FP64)
    p._fbuf, p._fbuf_lock, h = None, g._fbuf_lock, C.c_void_p()
    assert p.L.mdx_open(C.byref(p.packed.dims), C.byref(h)) == 0
    p.h = h
    p._check(p.L.mdx_set_params(h, C.byref(p.packed.params)))
    p._check(p.L.mdx_upload_topology(h, C.byref(p.packed.topo)))
    assert _same(a, _evaluate(p, st))
    g.close()
    p.close()


def test_tables_are_made_when_they_change():
    """The same parameters again launch nothing; another alpha or RSHORT and back
    gives what a context with them from the start gives."""
    from mdynamix_gb300.mdx import ForcePath
    s = _ions(150, 30.0, fexp=4.0)
    st = S.make_configuration(s, seed=4, jitter=0.05)
    g = ForcePath(s, precision=MDX_FP64)
    a = _evaluate(g, st)
    n = g.launches
    g.set_params(g.packed.params)
    assert g.launches == n
    assert _same(a, _evaluate(g, st))
    for change in (dict(alpha=3.0), dict(rshort=6.5), dict(rcut=8.5), {}):
        t = S.System(dataclasses.replace(s.spec, **change))
        f = ForcePath(t, precision=MDX_FP64)
        g.set_params(f.packed.params)
        assert _same(_evaluate(f, st), _evaluate(g, st)), change
        f.close()
    g.close()

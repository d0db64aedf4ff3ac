"""INIFUR when the device memory ends part-way (one of its allocations is refused by
the library's own hook, on the host): the FP64 path goes on with the FP64-pipe
passes where only the fixed-point passes' images found no room; otherwise the call
fails, and the next one starts over.  Forces against a context without refusals,
to the 1e-12 that test_ewald_fixed_point.py holds between the passes."""
import numpy as np
import pytest

from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED
from tests import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
def test_refused_allocations(prec):
    from mdynamix_gb300.mdx import ForcePath, MdxError
    s, st = systems.build(systems.spcfw(n=216))
    g = ForcePath(s, precision=prec)
    g.set_state(*st)
    g.chcnb()
    g.getcom()
    g.slforces()
    want = g.forces(2)
    g.close()
    tol = 1e-12 if prec == MDX_FP64 else 1e-5
    outcomes = []
    for k in range(1, 40):
        g = ForcePath(s, precision=prec)
        g.set_state(*st)
        g.chcnb()
        g.getcom()
        assert g.L.mdx_probe_fail_alloc(g.h, k) == 0
        try:
            g.slforces()
            outcomes.append("ok")
        except MdxError:
            outcomes.append("refused")
            g.slforces()
        f = g.forces(2)
        assert np.abs(f - want).max() <= tol * np.abs(f).max(), k
        if prec == MDX_FP64 and g.path_info()["ewald_force_pass"] == 0:
            outcomes[-1] += ", FP64 pipe"
        assert g.L.mdx_probe_fail_alloc(g.h, 0) == 0
        g.set_params(g.packed.params)  # a k-set again, all of it this time
        g.slforces()
        f = g.forces(2)
        assert np.abs(f - want).max() <= tol * np.abs(f).max(), k
        g.close()
    assert "refused" in outcomes and outcomes[-1] == "ok"  # past the last allocation
    assert prec == MDX_MIXED or "ok, FP64 pipe" in outcomes


def test_fixed_point_passes_cost_one_allocation(monkeypatch):
    """INIFUR with the fixed-point passes allocates no more often than with the
    FP64-pipe passes (an allocation waits for the stream).  Counted with the hook:
    the first allocation whose refusal changes nothing is one too many."""
    from mdynamix_gb300.mdx import ForcePath, MdxError
    s, st = systems.build(systems.spcfw(n=216))
    count = {}
    for tc, passes in (("0", 0), ("1", 3)):
        monkeypatch.setenv("MDX_EWALD_TC", tc)
        for k in range(1, 60):
            g = ForcePath(s, precision=MDX_FP64)
            assert g.L.mdx_probe_fail_alloc(g.h, k) == 0
            try:
                g.inifur()
                done = g.path_info()["ewald_force_pass"] == passes
            except MdxError:
                done = False
            g.close()
            if done:
                break
        count[tc] = k - 1
    assert 0 < count["1"] <= count["0"]

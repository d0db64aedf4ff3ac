"""SHEJK leaves a bond whose length is not a number alone, as ABS(DIFFSQ) > TOLER
does (mdstep.f:1180): the other molecules converge in the sweeps they need, none
counts as failed, and the step reports a non-finite value."""
import numpy as np
import pytest

from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED
from tests import systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [MDX_FP64, MDX_MIXED])
def test_not_a_number(prec):
    from mdynamix_gb300.mdx import ForcePath, MdxError
    s, st = systems.build(systems.spce_ions(n=60, ions=1, toler=1e-4))
    g = ForcePath(s, precision=prec)
    g.set_state(*st)
    g.sultan(1)  # lists and forces of the finite start
    xv, th = g.get_state()
    sweeps = g.sultan_steps(1, 1)[0].shake_iter
    assert 1 < sweeps < 100
    bad = [a.copy() for a in xv]
    bad[1][3 * 7] = np.nan  # the oxygen of one water
    g.set_state(*bad, thermo=th)
    with pytest.raises(MdxError, match="non-finite"):
        g.sultan_steps(1, 1)
    _, th = g.get_state()
    assert th.shake_fail == 0
    assert th.shake_iter_max <= sweeps
    g.close()

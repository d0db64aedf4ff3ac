"""mdx_get_path_info names the Ewald passes that run: the FP64 path's fixed-point
passes, its FP64-pipe passes when asked for or when the k-set does not fit, the
mixed path's."""
import pytest

from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tc,boz,passes", [
    (MDX_FP64, None, 20.0, (3, 3)), (MDX_FP64, "0", 20.0, (0, 0)),
    (MDX_FP64, None, 70.0, (0, 0)),  # |nz| past 31
    (MDX_MIXED, None, 20.0, (2, 1)), (MDX_MIXED, "0", 20.0, (1, 1)),
    (MDX_MIXED, "2", 20.0, (2, 2))])
def test_ewald_passes(prec, tc, boz, passes, monkeypatch):
    from mdynamix_gb300.mdx import ForcePath
    monkeypatch.setenv("MDX_EWALD_TC", tc) if tc else monkeypatch.delenv("MDX_EWALD_TC", False)
    s = S.System(S.RunSpec(molecules=[("SPC-FW", 40)], box=(13.0, 13.0, boz), dt_fs=2.0, nfreq=1,
                           rcut=5.5, rshort=5.0, alpha=0.35 * 5.5, fexp=16.0, ichnb=10,
                           trtemp=300.0))
    g = ForcePath(s, precision=prec)
    g.set_state(*S.make_configuration(s, seed=3, jitter=0.05))
    assert g.path_info()["sfac_slices"] == 0  # no k-set yet
    g.inifur()
    info = g.path_info()
    assert (info["ewald_force_pass"], info["ewald_sfac_pass"]) == passes
    assert info["sfac_slices"] >= 1 and info["sfac_ordered"] == 1
    g.close()

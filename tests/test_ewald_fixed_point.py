"""The FP64 path's reciprocal Ewald passes in fixed point on the tensor cores
(ewald_fx.cu) against the FP64-pipe passes (MDX_EWALD_TC=0) at the edges of
their tiles: atom counts around 32 and 128, K = 2 kz around 16, 48 and 64, X
and Y rows in and out of shared memory, the three cells, and k-sets past the
limits, where both runs are the FP64-pipe passes.

Tolerance: each operand carries 55 fractional bits and the class sums are
exact, so a force component is off by a few 2^-53 of the sum of its terms'
magnitudes; the FP64-pipe passes round each of up to 2 x 10^4 terms to 2^-53.
Both stay within 1e-13 of the largest force; 1e-12 is held."""
import numpy as np
import pytest

from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64

TOL = 1e-12


def _system(nwater, nion, box, cutk, icell=0):
    """Water and ion pairs with alpha 0.35 / A and k-vectors up to cutk (1 / A)."""
    rc = 5.5
    return S.System(S.RunSpec(
        molecules=[m for m in (("SPC-FW", nwater), ("Na+", nion), ("Cl-", nion)) if m[1]],
        box=box, dt_fs=2.0, nfreq=1, rcut=rc, rshort=5.0, alpha=0.35 * rc,
        fexp=cutk ** 2 / (4 * 0.35 ** 2), ichnb=10, trtemp=300.0, icell=icell))


def _slow(s, st, monkeypatch, tc):
    from mdynamix_gb300.mdx import ForcePath
    if tc is None:
        monkeypatch.delenv("MDX_EWALD_TC", raising=False)
    else:
        monkeypatch.setenv("MDX_EWALD_TC", tc)
    g = ForcePath(s, precision=MDX_FP64, nkv_max=400000)
    g.set_state(*st)
    g.chcnb()
    g.getcom()
    sc = g.slforces()
    f = g.forces(2)
    g.close()
    return sc, f


CASES = [
    # (waters, ion pairs, box, k cutoff, cell)
    (1, 1, (12.0, 12.0, 12.0), 1.6, 0),       # 5 atoms, K = 16
    (10, 0, (14.0, 14.0, 14.0), 3.0, 0),      # 30
    (10, 1, (14.0, 14.0, 14.0), 3.0, 0),      # 32
    (11, 0, (14.0, 14.0, 14.0), 3.1, 0),      # 33
    (42, 1, (16.0, 16.0, 16.0), 2.7, 0),      # 128
    (43, 0, (16.0, 17.0, 18.0), 2.7, 0),      # 129, unequal edges
    (341, 1, (23.0, 23.0, 23.0), 2.5, 0),     # 1025
    (100, 2, (20.0, 20.0, 50.0), 2.7, 0),     # kz 23: K = 48
    (100, 2, (20.0, 20.0, 53.0), 2.9, 0),     # kz 26: K = 64, X and Y rows in shared memory
    (100, 2, (44.0, 44.0, 44.0), 3.4, 0),     # kz 25, 50 rows: rows from global memory
    (100, 2, (44.0, 44.0, 40.0), 3.4, 0),     # K = 48, 50 rows: rows from global memory
    (40, 1, (13.0, 13.0, 70.0), 2.8, 0),      # kz 33: past K = 64
    (256, 2, (22.0, 22.0, 22.0), 2.5, 2),     # hexagonal
    (128, 2, (22.0, 22.0, 22.0), 2.2, 1),     # truncated octahedron
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=[f"{3 * c[0] + 2 * c[1]}-{c[2][2]:.0f}-{c[4]}" for c in CASES])
def test_fixed_point_ewald_matches_fp64_passes(case, monkeypatch):
    nw, ni, box, cutk, icell = case
    s = _system(nw, ni, box, cutk, icell)
    st = S.make_configuration(s, seed=3, jitter=0.05)
    a, fa = _slow(s, st, monkeypatch, "0")
    b, fb = _slow(s, st, monkeypatch, None)
    assert np.abs(fb - fa).max() <= TOL * np.abs(fa).max()
    for n in ("pels1", "qpe", "spe", "virx", "viry", "virz"):
        x, y = getattr(a, n), getattr(b, n)
        # the scalars sum terms of both signs: held to the largest of the energies
        assert abs(x - y) <= TOL * max(abs(a.qpe), abs(a.pels1), abs(x)), (n, x, y)


@pytest.mark.gpu
def test_fixed_point_ewald_reports_non_finite_positions(monkeypatch):
    """A non-finite coordinate makes S(k), the energy and the slow forces
    non-finite, as in the FP64-pipe passes."""
    s = _system(20, 1, (16.0, 16.0, 16.0), 2.5)
    st = list(S.make_configuration(s, seed=3, jitter=0.05))
    ref, _ = _slow(s, st, monkeypatch, None)
    assert np.isfinite(ref.qpe)
    from mdynamix_gb300.mdx import ForcePath
    g = ForcePath(s, precision=MDX_FP64)
    g.set_state(*st)
    g.chcnb()
    g.getcom()
    bad = [c.copy() for c in st]
    bad[2][7] = np.nan
    g.set_state(*bad)  # lists of the finite start
    sc = g.slforces()
    assert not np.isfinite(sc.qpe)
    assert not np.isfinite(g.forces(2)).any()
    g.set_state(*st)   # and back
    assert g.slforces().qpe == ref.qpe


@pytest.mark.gpu
def test_coherent_phases():
    """S(k) of atoms whose phases and charges are alike, the most that the digit
    sums can be asked to hold: 17,536 atoms of one sign in a row, and as many of the
    other with the same z spread among neutral ones, so that the two halves fill the
    sums to different heights and cancel.  The only k-vector is (0, 0, 1).

    Charges of 39 bits and the images' 55-bit phases are exact, so S(k) is 0 but for
    the rounding of each block's sum to the unit 2^-46 of 40,960 atoms: half a unit
    from at most 200 blocks, in either component."""
    import copy
    from mdynamix_gb300.mdx import ForcePath
    rng = np.random.default_rng(7)
    box, dense, n = (600.0, 600.0, 1500.0), 17536, 40960
    cutk = 1.5 * 2.0 * np.pi / box[2]
    s = S.System(S.RunSpec(molecules=[("Na+", n)], box=box, dt_fs=2.0, nfreq=1, rcut=25.0,
                           rshort=4.0, alpha=0.35 * 25.0, fexp=cutk ** 2 / (4 * 0.35 ** 2),
                           ichnb=10, trtemp=300.0))
    s = copy.copy(s)

    def digits(count, m):  # 0.d0 d1 .. in signed base 256 with d0 .. from 116 to 127
        d = rng.integers(116, 128, (count, m)).astype(float)
        return (d * 2.0 ** (-7.0 - 8.0 * np.arange(m))).sum(axis=1)

    q = digits(dense, 5)
    z = np.arccos(digits(dense, 6)) * box[2] / (2 * 3.1415926536) * rng.choice([-1.0, 1.0], dense)
    grid = rng.permutation(207 * 207)[:n]
    x, y = ((grid // 207 + 0.5) / 207 - 0.5) * box[0], ((grid % 207 + 0.5) / 207 - 0.5) * box[1]
    qs, zs = np.zeros(n), rng.uniform(-80.0, 80.0, n)
    qs[:dense], zs[:dense] = q, z
    other = (dense + np.arange(n - dense))[np.arange(n - dense) % 4 != 3][:dense]
    zs[other] = z
    s.site_charge = np.array([1.0])
    sums = []
    for sign in (0.0, -1.0):
        qs[other] = sign * q
        s.q = qs.copy()
        g = ForcePath(s, precision=MDX_FP64)
        g.set_state(x, y, zs, *[np.zeros(n)] * 3)
        g.chcnb()
        sc = g.slforces()
        assert sc.nkv == 1 and g.path_info()["ewald_sfac_pass"] == 3
        sums.append(sc.qpe)
        g.close()
    one = np.hypot((q * np.cos(2 * 3.1415926536 / box[2] * z)).sum(),
                   (q * np.sin(2 * 3.1415926536 / box[2] * z)).sum())
    assert np.sqrt(sums[1] / sums[0]) * one <= 200 * 2.0 ** -47 * np.sqrt(2.0)

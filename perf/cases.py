"""The work that users of this framework have it do, as cases that can be timed.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a user's program holds before the call (a context with
topology, parameters, start state and, for force calls, neighbour lists),
``run`` is one pass through the public entry points of
``mdynamix_gb300.mdx``, ``work`` the bytes and operations of a pass and
``exact`` the plain 64-bit answer where one is at hand (water forces).

Kinds of case:

* ``double``  a segment of the double time step loop from a restart state:
  upload, DOUBLE (its prologue with a list build, then long steps with their
  records, a list refresh every ten), download;
* ``sultan``  the same with SULTAN: leap-frog, SHAKE, in the bilayer with the
  anisotropic barostat;
* ``slow``    SLFORCES and its forces: the long-range half of a step, for a
  program that integrates by itself;
* ``all``     ALLFORCE and its forces: every force of a configuration;
* ``job``     a coupling state of an expanded-ensemble solvation job: RECINT,
  upload, a DOUBLE segment, the energy differences of a move, download;
* ``pimd``    long steps of a ring-polymer ensemble.

The mixed path computes forces in 32 bits (2e-6 of the 64-bit forces), and
trajectories are written as REAL*4, so what it returns is taken in float32;
the FP64 path's outputs stay float64.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from mdynamix_gb300 import system as S
from mdynamix_gb300.abi import MDX_FP64, MDX_MIXED
from mdynamix_gb300.mdx import ForcePath, PimdPath

# per listed pair, per (paired k record, atom), per (column, atom), per
# (phase-table row, atom): operations of the force expressions
OPS_PAIR, OPS_EW_PAIR, OPS_EW_COL, OPS_EW_ROW = 80, 24, 23, 8


def listed():
    return [
        # the benchmark: 98,304 atoms of flexible water, FP64 drop-in, one
        # list period of long steps (a production run is many of these)
        dict(name="fp64-double-98k", kind="double", prec="fp64", nwater=32768, steps=10),
        # the same run on the mixed path: what large runs use
        dict(name="mixed-double-98k", kind="double", prec="mixed", nwater=32768, steps=20),
        # one long-range force evaluation at that size, both paths: a program
        # with its own integrator, or an energy evaluation of a stored frame
        dict(name="fp64-slow-98k", kind="slow", prec="fp64", nwater=32768),
        dict(name="mixed-slow-98k", kind="slow", prec="mixed", nwater=32768),
        # an ordinary box: 1000 waters, Rc 9 A
        dict(name="fp64-double-3k", kind="double", prec="fp64", nwater=1000, steps=20),
        # all forces of a middle-sized box, an odd count of molecules
        dict(name="fp64-all-21k", kind="all", prec="fp64", nwater=7001),
        # the smallest call: a 600-atom box driven force call by force call
        dict(name="mixed-all-600", kind="all", prec="mixed", nwater=203),
        # serving: a small mixed job and a large FP64 one
        dict(name="mixed-job-600", kind="job", prec="mixed", solute="C2H5OH", nwater=211, steps=20),
        dict(name="fp64-job-6k", kind="job", prec="fp64", solute="dmso", nwater=1999, steps=10),
        # path integrals: 256 waters x 32 beads, mixed
        dict(name="mixed-pimd-32x768", kind="pimd", prec="mixed", nwater=256, nbeads=32, steps=40),
        # lipid bilayer, NPT, SHAKE on bonds to hydrogen, mixed
        dict(name="mixed-bilayer-22k", kind="sultan", prec="mixed", system="bilayer", steps=10),
        # rigid water and ions, SHAKE, FP64: the plain-method case
        dict(name="fp64-spce-1544", kind="sultan", prec="fp64", system="spce", nwater=512, steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["double", "double", "slow", "slow", "all", "job", "sultan", "pimd"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "double":
        return dict(kind=kind, prec=prec, nwater=_log(rng, 200, 32000), steps=rng.randint(2, 10))
    if kind in ("slow", "all"):
        return dict(kind=kind, prec=prec, nwater=_log(rng, 200, 32000))
    if kind == "job":
        return dict(kind=kind, prec=prec, solute=rng.choice(S.SOLUTES),
                    nwater=_log(rng, 200, 2000), steps=rng.randint(5, 20))
    if kind == "sultan":
        return dict(kind=kind, prec=prec, system="spce", nwater=_log(rng, 400, 2000),
                    steps=rng.randint(5, 20))
    return dict(kind=kind, prec=prec, nwater=_log(rng, 200, 400), nbeads=rng.choice([4, 8, 16, 32]),
                steps=rng.randint(5, 20))


# ------------------------------------------------------------------ systems --
@functools.lru_cache(maxsize=8)
def _system(kind, name, nwater, nbeads, solute):
    """Topology and tables: read once by a program, whatever its start."""
    if kind == "job":
        spec = S.solvation_job(solute, nwater)
    elif kind == "pimd":
        spec = S.pimd_water(nwater=nwater, nbeads=nbeads)
    elif name == "bilayer":
        spec = S.dmpc_bilayer(shake_hbonds=True)
    elif name == "spce":
        # TOLER is squared by SHEJK: 1.4e-4 asks for 1e-8 of a bond length
        spec = dataclasses.replace(S.spce_nacl_nve(nwater=nwater), toler=1.4e-4, nvt=(300.0, 30.0))
    elif nwater >= 4000:
        # Rc 12 A, Ewald 0.25 / A, |n| growing with the box to 20 at 32,768
        spec = S.spcfw_water(nwater=nwater, nmax=max(4, round(20 * (nwater / 32768) ** (1 / 3))))
    else:
        rc = 9.0 if nwater >= 200 else 7.0
        spec = S.RunSpec(molecules=[("SPC-FW", nwater)], density=1.0, dt_fs=2.0, nfreq=10,
                         rcut=rc, rshort=5.0, alpha=2.8, fexp=12.0, ichnb=10,
                         nvt=(300.0, 30.0), trtemp=300.0)
    return S.System(spec)


def _sys(case):
    return _system(case["kind"], case.get("system", "water"), case.get("nwater", 0),
                   case.get("nbeads", 1), case.get("solute", ""))


# SPC-FW: sites O, H, H (A, amu, e)
_W_R = np.array([[0.0, 0.0, -0.0623071727522009], [0.0, -0.8451, 0.49448282724779913],
                 [0.0, 0.8451, 0.49448282724779913]])
_W_M = np.array([15.9994, 1.008, 1.008])


def _water_box(nwater, box, seed):
    """Positions [3 nwater, 3]: molecules at random orientations on a jittered
    cubic lattice, as a freshly built box."""
    rng = np.random.default_rng(seed)
    side = int(math.ceil(nwater ** (1.0 / 3.0) - 1e-9))
    a = box / side
    cell = rng.permutation(side ** 3)[:nwater]
    com = np.stack([cell // (side * side), (cell // side) % side, cell % side], 1)
    com = (com + 0.5) * a - 0.5 * box + rng.uniform(-0.05, 0.05, (nwater, 3)) * a
    q = rng.normal(size=(nwater, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                    2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                    2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)],
                   1).reshape(nwater, 3, 3)
    pos = np.einsum("nij,sj->nsi", rot, _W_R) + com[:, None, :]
    return pos.reshape(-1, 3), rng


def _momenta(s, rng):
    """Maxwell momenta at the target temperature, no net drift."""
    v = rng.normal(size=(3, s.nstot)) / np.sqrt(s.massdi)
    v -= v.sum(axis=1, keepdims=True) / s.nstot
    temp = 1.5 * float((v * v * s.massdi).sum()) * s.enerf * s.tempf / s.fnst
    return list(v * math.sqrt(s.trtemp / temp))


@functools.lru_cache(maxsize=2)
def _bilayer_start():
    """The packed bilayer (a stored start); the seed gives the momenta and a
    thermal jitter."""
    return S.bilayer_configuration(_system("sultan", "bilayer", 0, 1, ""), seed=1)


def _start(case, s, seed):
    if case["kind"] in ("double", "slow", "all"):
        pos, rng = _water_box(case["nwater"], s.boxl, seed)
        return [np.ascontiguousarray(c) for c in pos.T] + _momenta(s, rng)
    if case.get("system") == "bilayer":
        st = _bilayer_start()
        rng = np.random.default_rng(seed)
        return [c + rng.normal(size=s.nstot) * 0.003 for c in st[:3]] + _momenta(s, rng)
    return list(S.make_configuration(s, seed=seed, jitter=0.05))


def prepare(case, seed):
    s = _sys(case)
    prec = MDX_FP64 if case["prec"] == "fp64" else MDX_MIXED
    if case["kind"] == "pimd":
        g = PimdPath(s, S.pimd_beads(s, seed=seed), precision=prec)
        g.run(0)
        return dict(case=case, path=g, mstep=0)
    st = _start(case, s, seed)
    g = ForcePath(s, precision=prec)
    if case["kind"] in ("slow", "all"):
        g.set_state(*st)
        g.chcnb()
        g.getcom()
    return dict(case=case, path=g, start=st)


# ---------------------------------------------------------------------- run --
_REC = ("pe1", "pels1", "pe2", "pels2", "spe", "pint", "tke", "temp")


def _records(recs, dt, names=_REC):
    return {n: np.array([getattr(r, n) for r in recs], dt) for n in names}


def run(state):
    case, g = state["case"], state["path"]
    kind = case["kind"]
    dt = np.float64 if case["prec"] == "fp64" else np.float32
    if kind in ("slow", "all"):
        sc = g.slforces() if kind == "slow" else g.allforce()
        f = g.forces(2 if kind == "slow" else 3)
        names = ("pe1", "pels1", "spe", "virx", "viry", "virz")
        if kind == "all":
            names += ("pe2", "pels2", "pint")
        return {"forces": f.astype(dt, copy=False), **{n: dt(getattr(sc, n)) for n in names}}
    if kind == "pimd":
        recs = g.steps(case["steps"], state["mstep"])
        state["mstep"] += case["steps"]
        return {"beads": np.asarray(g.states(), dt),
                **_records(recs, dt, ("qek", "pe", "tke", "temp"))}
    out = {}
    if kind == "job":
        g.set_lambda(0.5)
    g.set_state(*state["start"])
    recs = g.sultan(case["steps"]) if kind == "sultan" else g.double(case["steps"])
    if kind == "job":
        out["move"] = np.array(g.ee_delta(0.5, 0.25), dt)
    xv, th = g.get_state()
    out.update(state=[a.astype(dt, copy=False) for a in xv],
               box=np.array([th.boxl, th.boyl, th.bozl], dt), **_records(recs, dt))
    return out


# --------------------------------------------------------------------- work --
def work(case):
    s = _sys(case)
    n, rho = s.nstot, s.nstot / s.vol
    pairs = lambda r0, r1: n * rho * 2.0 / 3.0 * math.pi * (r1 ** 3 - r0 ** 3)  # noqa: E731
    rs = s.spec.rshort
    short, long_ = OPS_PAIR * pairs(0.0, rs), OPS_PAIR * pairs(rs, s.rcutt)
    ncol, npair, rows = s.kcolumn_counts()
    ew = (OPS_EW_PAIR * npair + OPS_EW_COL * ncol + OPS_EW_ROW * rows) * n
    xv = 48 * n  # positions and momenta, each way
    kind = case["kind"]
    if kind == "slow":
        return {"bytes": 56 * n, "flops": long_ + ew}
    if kind == "all":
        return {"bytes": 56 * n, "flops": short + long_ + ew}
    step = s.spec.nfreq * short + long_ + ew
    if kind == "pimd":
        return {"bytes": case["nbeads"] * (xv + 2 * 48 * n * case["steps"]),
                "flops": case["nbeads"] * case["steps"] * step}
    # the state crosses the host link once each way and HBM once a short step
    return {"bytes": 2 * xv + 2 * xv * s.spec.nfreq * case["steps"],
            "flops": (case["steps"] + 1) * step}


# -------------------------------------------------------------------- exact --
# SPC-FW and the units of the reference's input (its own literals)
_AVSNO, _ELECHG, _EPS0, _PI = 6.02252e23, 1.602e-19, 8.854e-12, 3.1415926536
_ERFC = (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429, 0.3275911)
_TOTPI = 1.128379169


def _erfc_terms(alpha, r):
    """The reference's erfc polynomial and exp(-(alpha r)^2)."""
    a1, a2, a3, a4, a5, b1 = _ERFC
    ar = alpha * r
    t = 1.0 / (1.0 + b1 * ar)
    e = torch.exp(-ar * ar)
    return ((((a5 * t + a4) * t + a3) * t + a2) * t + a1) * t * e, e


def exact(case, seed):
    """Water forces and energies in 64 bits: every pair, every k-vector."""
    if case["kind"] not in ("slow", "all"):
        return None
    nw = case["nwater"]
    n = 3 * nw
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    # the box of 1 g/cm3 and the run parameters of _system
    tot = 18.0154 * nw / (_AVSNO * 1000.0)
    vol = _AVSNO / float(nw) * (tot / 1000.0) * nw * 1e30 / _AVSNO
    box = vol ** (1.0 / 3.0)
    if nw >= 4000:
        rc, alpha_in = 12.0, 3.0
        nmax = max(4, round(20 * (nw / 32768) ** (1 / 3)))
        side = (nw * (15.9994 + 2 * 1.008) / (_AVSNO * 1000.0) / 1000.0 * 1e30) ** (1.0 / 3.0)
        fexp = math.ceil((2 * _PI * nmax / side) ** 2 / (4 * 0.25 ** 2) * 100.0) / 100.0
    else:
        rc, alpha_in, fexp = (9.0 if nw >= 200 else 7.0), 2.8, 12.0
    alpha = alpha_in / rc if rc <= 0.5 * box else 2.0 * alpha_in / box
    unite = tot * (1e-10 / 2e-15) ** 2
    coulf = (_ELECHG / _EPS0) * (_ELECHG / unite) / (4.0 * _PI * 1e-10)
    efact = 1e3 / _AVSNO / unite
    a6 = -4.0 * 0.6502 * efact * 3.1656 ** 6
    b12 = 4.0 * 0.6502 * efact * 3.1656 ** 12
    pos = torch.tensor(_water_box(nw, box, seed)[0], **f64)
    q = torch.tensor([-0.82, 0.41, 0.41], **f64).repeat(nw)
    mol = torch.arange(n, device=dev) // 3
    oxy = torch.arange(n, device=dev) % 3 == 0
    force = torch.zeros(n, 3, **f64)
    e = dict.fromkeys(("pe1", "pels1", "pe2", "pels2"), 0.0)
    half = 0.5 * box

    def image(d):
        return torch.where(d.abs() > half, d - torch.copysign(torch.full_like(d, box), d), d)

    step = max(16, min(n, 100_000_000 // n))
    for i0 in range(0, n, step):  # rows of atoms against all atoms
        i1 = min(n, i0 + step)
        rr = torch.zeros(i1 - i0, n, **f64)
        for a in range(3):
            rr += image(pos[i0:i1, a, None] - pos[None, :, a]) ** 2
        keep = (rr <= rc * rc) & (mol[i0:i1, None] != mol[None, :])
        ii, jj = torch.nonzero(keep, as_tuple=True)
        r2 = rr[ii, jj]
        del rr, keep
        ii = ii + i0
        d = image(pos[ii] - pos[jj])
        r = torch.sqrt(r2)
        erfc, ex = _erfc_terms(alpha, r)
        e1 = coulf * q[ii] * q[jj] / r
        f = e1 * (_TOTPI * alpha * ex + erfc / r) / r
        lj = (oxy[ii] & oxy[jj]).to(torch.float64)
        r6 = lj / r2 ** 3
        esr = (a6 + b12 * r6) * r6
        f = f + (6.0 * a6 + 12.0 * b12 * r6) * r6 / r2
        near = r2 <= 25.0
        if case["kind"] == "slow":
            f = torch.where(near, torch.zeros_like(f), f)
        force.index_add_(0, ii, f[:, None] * d)
        e["pels2"] += 0.5 * float((e1 * erfc)[near].sum())
        e["pe2"] += 0.5 * float(esr[near].sum())
        e["pels1"] += 0.5 * float((e1 * erfc)[~near].sum())
        e["pe1"] += 0.5 * float(esr[~near].sum())
    # reciprocal space: half of the k sphere
    alp2 = alpha * alpha
    cutk2 = 4.0 * alp2 * fexp
    kmax = int(math.sqrt(cutk2) * box / (2 * _PI) + 1)
    th = pos * (2 * _PI / box)
    ns = torch.arange(-kmax, kmax + 1, **f64)
    tz = torch.exp(1j * th[:, 2:3] * ns)  # [n, 2 kmax + 1]
    ty = torch.exp(1j * th[:, 1:2] * ns)
    two = 2 * _PI / box
    for ix in range(0, kmax + 1):
        t = (q * torch.exp(1j * ix * th[:, 0]))[:, None] * ty  # charge and x, y phases
        sk = t.transpose(0, 1) @ tz
        rk2 = two * two * (ix * ix + ns[:, None] ** 2 + ns[None, :] ** 2)
        use = rk2 <= cutk2
        if ix == 0:
            use &= (ns[:, None] > 0) | ((ns[:, None] == 0) & (ns[None, :] > 0))
        akc = torch.where(use, 4.0 * _PI * coulf / box ** 3 * torch.exp(-0.25 * rk2 / alp2)
                          / torch.where(use, rk2, torch.ones_like(rk2)), torch.zeros_like(rk2))
        e["pels1"] += float((akc * (sk.real ** 2 + sk.imag ** 2)).sum())
        w = 2.0 * akc * sk.conj()
        u = t * (tz @ w.transpose(0, 1))
        v = t * (tz @ (w * (two * ns)[None, :]).transpose(0, 1))
        force[:, 0] += two * ix * u.imag.sum(1)
        force[:, 1] += (u.imag * (two * ns)).sum(1)
        force[:, 2] += v.imag.sum(1)
        del t, u, v
    # excluded pairs of a molecule, self energy
    p = pos.reshape(nw, 3, 3)
    fm = force.reshape(nw, 3, 3)
    qs = (-0.82, 0.41, 0.41)
    spe = -alpha / math.sqrt(_PI) * coulf * nw * (0.82 ** 2 + 2 * 0.41 ** 2)
    for a, b in ((0, 1), (0, 2), (1, 2)):
        d = image(p[:, a] - p[:, b])
        r2 = (d * d).sum(1)
        r = torch.sqrt(r2)
        erfc, ex = _erfc_terms(alpha, r)
        qij = coulf * qs[a] * qs[b]
        spe += float((qij * (erfc - 1.0) / r).sum())
        f = (qij * (_TOTPI * alpha * r * ex + erfc - 1.0) / (r * r2))[:, None] * d
        fm[:, a] += f
        fm[:, b] -= f
    out = {"spe": spe, "virx": None, "viry": None, "virz": None}
    names = ("pe1", "pels1")
    if case["kind"] == "all":  # harmonic bonds and angle
        names += ("pe2", "pels2")
        pint = 0.0
        for h in (1, 2):
            d = image(p[:, h] - p[:, 0])
            r = torch.sqrt((d * d).sum(1))
            pint += float((2217.0 * efact * (r - 1.012) ** 2).sum())
            f = (-2.0 * 2217.0 * efact * (r - 1.012) / r)[:, None] * d
            fm[:, h] += f
            fm[:, 0] -= f
        u, v = image(p[:, 1] - p[:, 0]), image(p[:, 2] - p[:, 0])
        u2, v2 = (u * u).sum(1), (v * v).sum(1)
        uv = torch.sqrt(u2 * v2)
        cos = (u * v).sum(1) / uv
        phi = torch.acos(cos)
        dphi = phi - 113.24 / (180.0 / _PI)
        pint += float((158.9 * efact * dphi ** 2).sum())
        s = (-2.0 * 158.9 * efact * dphi / torch.sin(phi))[:, None]
        fu = s * (v / uv[:, None] - cos[:, None] * u / u2[:, None])
        fv = s * (u / uv[:, None] - cos[:, None] * v / v2[:, None])
        fm[:, 1] -= fu
        fm[:, 2] -= fv
        fm[:, 0] += fu + fv
        out["pint"] = pint
    out.update({k: e[k] for k in names})
    out = {k: None if v is None else np.float64(v) for k, v in out.items()}
    out["forces"] = fm.reshape(n, 3).cpu().numpy()
    return out

"""Performance cases of the structure-factor engine: what a user's program asks of it.

Every case is one call (or one batched submission, or one refinement cycle) through the public entry points of
``discamb_gb300.api``.  A case says

* ``model``: ``hc`` (Hansen-Coppens multipoles), ``iam`` (n-Gaussian form factors) or ``tab`` (tabulated form
  factors, Hirshfeld-atom style);
* ``group``, ``atoms``, ``hkl``, ``types``: the crystal (``types`` 0: every atom has its own multipole type);
* ``adp``: ``aniso`` (hydrogen atoms stay isotropic, as in refinements) or ``iso`` (isotropic B throughout);
* ``precision``: 64 (the plain FP64 form, the default of the calls) or 32 (the FP32-bulk form);
* ``want``: ``f`` (structure factors only), ``grad`` (with the derivatives by xyz, U and occupancy) or ``full``
  (with the multipole-parameter derivatives too);
* ``call``: ``host`` (atoms and dT/dF from host arrays, results in host arrays), ``device`` (device buffers on the
  caller's stream, resident atoms) or ``cycle`` (a multipole refinement cycle: new multipole parameters, new
  atoms, then the device call);
* ``count`` > 1: that many crystals of uneven size in one submission (``mix`` seeds their sizes and groups; the
  sizes are log-uniform up to ``atoms`` and ``hkl``).

The FP32-bulk form's results carry 24 bits in 64-bit buffers; a program that asks for that form keeps them as one
flat FP32 vector (what an optimiser on the GPU takes), and so do the cases.  FP64 results stay FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from discamb_gb300 import api
from discamb_gb300.crystal import space_group
from discamb_gb300.model import AtomType, Orbital, Structure, Wavefunction

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def _case(name, **kw):
    c = dict(name=name, model="hc", group="P212121", atoms=100, hkl=5000, types=0, adp="aniso", precision=32,
             want="grad", call="device", count=1, mix=0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest request of a refinement service: a small triclinic molecule, latency and launches only
        _case("molecule P-1 f32", group="P-1", atoms=20, hkl=1501),
        # the call a small-molecule refinement makes by default: FP64, host arrays in and out, P2_1/c
        _case("molecule P21/c f64 host", group="P21/c", atoms=32, hkl=4573, precision=64, call="host"),
        # charge-density refinement: multipole parameters and atoms change every cycle, all derivatives, FP64
        _case("charge density f64 cycle", atoms=64, hkl=16001, precision=64, want="full", call="cycle"),
        # the median request of the service: a mid-size centred monoclinic structure
        _case("organic C2/c f32", group="C2/c", atoms=633, hkl=17321, types=64),
        # a macromolecule with transferred multipoles (150 atom types), isotropic B
        _case("protein iso f32", atoms=5000, hkl=54704, types=150, adp="iso"),
        # the same model in the plain FP64 form, one screw axis
        _case("protein P21 f64", group="P21", atoms=2501, hkl=30011, types=100, precision=64, adp="iso"),
        # electron-density map coefficients: structure factors without derivatives
        _case("protein F only f32", atoms=8000, hkl=100003, types=150, want="f"),
        # the largest structure: 50,000 atoms, eight operations, the full derivative set
        _case("large full f32", group="P43212", atoms=50000, hkl=315281, types=300, want="full"),
        # the same derivative set in FP64 on a structure that FP64 is asked for
        _case("tetragonal full f64", group="P43212", atoms=1200, hkl=20011, types=100, precision=64, want="full"),
        # independent-atom refinement of a mid-size structure, all operations summed
        _case("iam P21/c f32", model="iam", group="P21/c", atoms=2000, hkl=50021, types=5),
        # Hirshfeld-atom refinement of one molecule in FP64 from a table of form factors
        _case("table P21/c f64", model="tab", group="P21/c", atoms=150, hkl=20021, precision=64),
        # a batch of Hirshfeld-atom refinements of uneven size: streams the tables from HBM
        _case("table batch f32", model="tab", group="P21/c", atoms=2000, hkl=100000, count=24, mix=4),
    ]


_GROUPS = ("P1", "P-1", "P21", "P21/c", "P212121", "C2/c", "P43212", "Pbca")
_MULT = {"P1": 1, "P-1": 2, "P21": 2, "P21/c": 4, "P212121": 4, "C2/c": 4, "P43212": 8, "Pbca": 8}


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any model, group, precision and call."""
    kind = rng.choice(["small", "small", "hc", "hc", "hc", "full", "fonly", "iam", "tab", "batch"])
    group = rng.choice(_GROUPS)
    precision = rng.choice([32, 64])
    cap = 1.5e10 if precision == 32 else 1.2e9  # terms: at most about a tenth of a second at the start
    if kind == "batch":
        model = rng.choice(["tab", "hc"])
        return _drawn(model=model, group="P21/c" if model == "tab" else "mixed",
                      atoms=_log_uniform(rng, 200, 2000), hkl=_log_uniform(rng, 10000, 60000),
                      types=0 if model == "tab" else 64, count=rng.randint(5, 20), mix=rng.randint(1, 1000))
    if kind == "small":
        atoms = _log_uniform(rng, 8, 200)
        return _drawn(group=group, atoms=atoms, hkl=_log_uniform(rng, 500, 150 * atoms + 1000), precision=precision,
                      call=rng.choice(["device", "host", "cycle"]), want=rng.choice(["grad", "grad", "full"]),
                      types=rng.choice([0, 10]))
    atoms = _log_uniform(rng, 100, 20000 if precision == 32 else 4000)
    if kind == "tab":
        atoms = min(atoms, 2000)
    hkl = _log_uniform(rng, 2000, max(4000, min(300000, 40 * atoms)))
    hkl = max(501, min(hkl, int(cap / (atoms * _MULT[group]))))
    return _drawn(model=kind if kind in ("iam", "tab") else "hc", group=group, atoms=atoms, hkl=hkl,
                  types={"iam": 5, "tab": 0}.get(kind, rng.randint(20, 200)), precision=precision,
                  adp=rng.choice(["aniso", "aniso", "iso"]),
                  want={"full": "full", "fonly": "f"}.get(kind, "grad"))


def _drawn(**kw):
    c = _case("", **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs (plain numpy, from the seed alone)
# ---------------------------------------------------------------------------
_BOHR = 0.529177
#            Z, occupancy core / valence, exponents (1/bohr) core / valence, powers core / valence, f' + i f"
_ELEMENT = {
    "H": (1, 0, 1, (), (1.0, 1.6), (), (0, 0), 0j),
    "C": (6, 2, 4, (5.4, 8.0), (1.6, 2.6), (0, 0), (1, 1), 0.0033 + 0.0016j),
    "N": (7, 2, 5, (6.4, 9.4), (1.9, 3.0), (0, 0), (1, 1), 0.0061 + 0.0033j),
    "O": (8, 2, 6, (7.4, 10.8), (2.2, 3.4), (0, 0), (1, 1), 0.0106 + 0.0060j),
    "S": (16, 10, 6, (14.0, 6.0), (1.8, 2.9), (0, 1), (2, 2), 0.1246 + 0.1234j),
}
_DEF_POW = {"H": [0, 1, 2], "C": [2, 2, 2, 3, 4], "N": [2, 2, 2, 3, 4], "O": [2, 2, 2, 3, 4], "S": [4, 4, 4, 4, 4]}
_SYMBOLS = "CHNOS"
_SHARE = np.array([0.32, 0.49, 0.085, 0.10, 0.005])
# Gaussians of the tabulated model's spherical part: Z sum_i w_i exp(-b_i s^2)
_F0_W = np.array([0.4, 0.3, 0.3])
_F0_B = {"H": (10.0, 25.0, 3.0), "C": (20.0, 8.0, 0.5), "N": (16.0, 6.5, 0.4), "O": (13.0, 5.0, 0.3),
         "S": (12.0, 4.0, 0.3)}

# operations the engine sums over: R (rows), translation; centrosymmetric groups of the HC model: the subset
# without the inversion (at the origin); C: the C-centring multiplier 2
_E, _2X, _2Y, _2Z = np.diag([1, 1, 1]), np.diag([1, -1, -1]), np.diag([-1, 1, -1]), np.diag([-1, -1, 1])
_R4 = np.array([[0, -1, 0], [1, 0, 0], [0, 0, 1]])
_SUBSET = {
    "P1": ([(_E, (0, 0, 0))], False),
    "P-1": ([(_E, (0, 0, 0))], True),
    "P21": ([(_E, (0, 0, 0)), (_2Y, (0, .5, 0))], False),
    "P21/c": ([(_E, (0, 0, 0)), (_2Y, (0, .5, .5))], True),
    "C2/c": ([(_E, (0, 0, 0)), (_2Y, (0, 0, .5))], True),
    "P212121": ([(_E, (0, 0, 0)), (_2Z, (.5, 0, .5)), (_2Y, (0, .5, .5)), (_2X, (.5, .5, 0))], False),
    "Pbca": ([(_E, (0, 0, 0)), (_2Z, (.5, 0, .5)), (_2Y, (0, .5, .5)), (_2X, (.5, .5, 0))], True),
    "P43212": ([(_E, (0, 0, 0)), (_2Z, (0, 0, .5)), (_R4, (.5, .5, .75)), (_R4.T, (.5, .5, .25)),
                (_2Y, (.5, .5, .75)), (_2X, (.5, .5, .25)), (np.array([[0, 1, 0], [1, 0, 0], [0, 0, -1]]), (0, 0, 0)),
                (np.array([[0, -1, 0], [-1, 0, 0], [0, 0, -1]]), (0, 0, .5))], False),
}


def _all_operations(group):
    ops, centro = _SUBSET[group]
    return ops + [(-r, tuple(-np.array(t))) for r, t in ops] if centro else ops


def _frac_to_cart(cell):
    a, b, c = cell[:3]
    ca, cb, cg = (math.cos(math.radians(v)) for v in cell[3:])
    sg = math.sin(math.radians(cell[5]))
    phi = math.sqrt(1 - ca * ca - cb * cb - cg * cg + 2 * ca * cb * cg)
    return np.array([[a, b * cg, c * cb], [0, b * sg, c * (ca - cb * cg) / sg], [0, 0, c * phi / sg]])


def _cell(group, n_atoms, rng):
    """A cell of 18 cubic Angstrom per atom of the group's crystal system."""
    ang = {"P1": (rng.uniform(80, 100), rng.uniform(95, 110), rng.uniform(80, 100))}
    ang["P-1"] = ang["P1"]
    for g in ("P21", "P21/c", "C2/c"):
        ang[g] = (90.0, rng.uniform(95, 110), 90.0)
    angles = ang.get(group, (90.0, 90.0, 90.0))
    r = rng.uniform(0.8, 1.25, 3)
    if group == "P43212":
        r[1] = r[0]
    centring = 2 if group == "C2/c" else 1
    v1 = abs(np.linalg.det(_frac_to_cart((*r, *angles))))
    edge = (18.0 * n_atoms * _MULT[group] * centring / v1) ** (1 / 3)
    return (*(edge * r), *angles)


def _reflections(group, cell, n):
    """The n lowest-angle unique reflections (000 and lattice absences left out)."""
    m = _frac_to_cart(cell)
    b = np.linalg.inv(m).T
    vol = abs(np.linalg.det(m))
    share = {"P1": 2, "P-1": 2, "P21": 4, "P21/c": 4, "C2/c": 8, "P43212": 16}.get(group, 8)
    r = (n * share * 1.15 / vol * 3 / (4 * math.pi)) ** (1 / 3) + 2.0 / vol ** (1 / 3)
    while True:
        lim = [int(r * np.linalg.norm(m[:, i])) + 1 for i in range(3)]
        low = [-lim[0] if share <= 4 or group == "C2/c" else 0, -lim[1] if share == 2 else 0, 0]
        g = np.meshgrid(*(np.arange(lo, hi + 1) for lo, hi in zip(low, lim)), indexing="ij")
        h = np.stack([v.ravel() for v in g], 1)
        keep = np.abs(h).sum(1) > 0
        h0, h1, h2 = h.T
        if share == 2:
            keep &= (h2 > 0) | (h0 > 0) | ((h0 == 0) & (h1 > 0))
        elif low[0] < 0:
            keep &= (h2 > 0) | (h0 >= 0)
        if group == "C2/c":
            keep &= (h0 + h1) % 2 == 0
        if group == "P43212":
            keep &= h0 >= h1
        h = h[keep]
        s = ((h @ b.T) ** 2).sum(1)
        inside = s <= r * r
        if inside.sum() >= n:
            h, s = h[inside], s[inside]
            return np.ascontiguousarray(h[np.argsort(s, kind="stable")[:n]].astype(np.int32))
        r *= 1.15


def _unit_norm(powers, exps, coeffs):
    s = sum(c * d * math.factorial(p + q + 2) / (a + b) ** (p + q + 3)
            for p, a, c in zip(powers, exps, coeffs) for q, b, d in zip(powers, exps, coeffs))
    return [c / math.sqrt(s) for c in coeffs]


def _inputs(case, seed, k=0, atoms=None, hkl=None, group=None):
    """Crystal k of a case as plain arrays."""
    group, n, m = group or case["group"], atoms or case["atoms"], hkl or case["hkl"]
    fixed = np.random.default_rng([case["mix"], k, n, m])  # the crystal: its cell and reflections
    rng = np.random.default_rng([seed, k])                 # the rest
    d = dict(group=group, cell=_cell(group, n, fixed))
    d["hkl"] = _reflections(group, d["cell"], m)
    el = rng.choice(5, n, p=_SHARE)
    el[:4] = [0, 1, 2, 3]
    d["element"] = el
    # wavefunctions, one per element: a core and a valence orbital of two Slater functions each
    d["wfn"] = []
    for sym in _SYMBOLS:
        z, occ_c, occ_v, ec, ev, pc, pv, anom = _ELEMENT[sym]
        orb = []
        for occ, ex, po in ((occ_c, ec, pc), (occ_v, ev, pv)):
            if ex:
                ex = [e / _BOHR * rng.uniform(0.95, 1.05) for e in ex]
                orb.append((occ, list(po), ex, _unit_norm(po, ex, [1.0, rng.uniform(0.2, 0.6)])))
        d["wfn"].append(dict(symbol=sym, z=z, orbitals=orb, zeta=rng.uniform(3, 5) / _BOHR, pow=_DEF_POW[sym],
                             anomalous=anom))
    # multipole types
    if case["types"] == 0 or case["model"] == "tab":
        d["type"], t_el = np.arange(n), el
    else:
        nt = max(5, min(case["types"], n))
        t_el = np.concatenate([np.arange(5), rng.choice(5, nt - 5, p=_SHARE)])
        d["type"] = np.zeros(n, dtype=np.int64)
        for e in range(5):
            own = np.nonzero(t_el == e)[0]
            d["type"][el == e] = own[rng.integers(len(own), size=int((el == e).sum()))]
    nt = len(t_el)
    d["type_element"] = t_el
    plm = rng.normal(0, 0.05, (nt, 25))
    plm[t_el == 1, 9:] = 0.0  # hydrogen: l <= 2
    d.update(plm=plm, n_l=np.where(t_el == 1, 3, 5), p_val=rng.uniform(3, 6, nt), kappa=rng.uniform(.9, 1.1, nt),
             kappa_p=rng.uniform(.9, 1.1, nt))
    # positions on a jittered grid, local frames, displacement parameters
    lengths = np.array(d["cell"][:3])
    grid = np.maximum(1, np.floor(lengths / (np.prod(lengths) / (1.3 * n)) ** (1 / 3)).astype(int))
    while grid.prod() < n:
        grid += 1
    at = rng.choice(grid.prod(), n, replace=False)
    d["xyz"] = (np.stack(np.unravel_index(at, tuple(grid)), 1) + 0.5 + rng.uniform(-.3, .3, (n, 3))) / grid
    q, r = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    q = q * np.sign(np.einsum("nii->ni", r))[:, None, :]
    q[np.linalg.det(q) < 0, :, 0] *= -1
    d["lcs"] = q
    iso = np.ones(n, bool) if case["adp"] == "iso" else el == 1
    qu = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    u = np.einsum("nik,nk,njk->nij", qu, rng.uniform(.01, .05, (n, 3)), qu)
    mm = _frac_to_cart(d["cell"])
    a = np.linalg.inv(mm @ np.diag(np.linalg.norm(np.linalg.inv(mm).T, axis=0)))  # U_cart -> U_cif
    u = np.einsum("ik,nkl,jl->nij", a, u, a)
    adp = np.stack([u[:, 0, 0], u[:, 1, 1], u[:, 2, 2], u[:, 0, 1], u[:, 0, 2], u[:, 1, 2]], 1)
    adp[iso] = 0.0
    uiso = rng.uniform(10, 40, n) / (8 * math.pi ** 2) if case["adp"] == "iso" else rng.uniform(.02, .06, n)
    adp[iso, 0] = uiso[iso]
    d.update(adp=adp, iso=iso, occupancy=rng.uniform(.8, 1.0, n), dtdf=rng.normal(size=m) + 1j * rng.normal(size=m))
    d["anomalous"] = np.array([_ELEMENT[s][7] for s in _SYMBOLS])[el]
    if case["model"] == "iam":
        d["iam"] = dict(ngauss=np.full(nt, 4, np.int32), a=rng.uniform(.5, 2.5, (nt, 5)),
                        b=rng.uniform(.5, 30, (nt, 5)), c=rng.uniform(0, .3, nt))
    return d


def _crystals(case, seed):
    if case["count"] == 1:
        return [_inputs(case, seed)]
    return [_inputs(case, seed, k, *size) for k, size in enumerate(_sizes(case))]


def _sizes(case):
    """(atoms, reflections, group) of every crystal."""
    if case["count"] == 1:
        return [(case["atoms"], case["hkl"], case["group"])]
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = int(math.exp(rng.uniform(math.log(10), math.log(case["atoms"]))))
        m = int(math.exp(rng.uniform(math.log(2000), math.log(case["hkl"]))))
        out.append((n, m, _GROUPS[int(rng.integers(6))] if case["group"] == "mixed" else case["group"]))
    return out


def _table(d, seed, k):
    """Tabulated form factors f0(|h|) (1 + 0.05 CN(0, 1)) on the device: complex64 [hkl][operation][atom]."""
    dev = "cuda"
    b = np.linalg.inv(_frac_to_cart(d["cell"])).T
    s2 = torch.tensor(((d["hkl"] @ b.T) ** 2).sum(1) * 0.25, device=dev)
    f0 = torch.stack([_ELEMENT[s][0] * sum(w * torch.exp(-x * s2) for w, x in zip(_F0_W, _F0_B[s]))
                      for s in _SYMBOLS], 1).float()[:, torch.tensor(d["element"], device=dev)]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed * 1009 + k)
    t = torch.randn((len(s2), len(_all_operations(d["group"])), len(d["xyz"]), 2), generator=gen, device=dev)
    t *= 0.05 / math.sqrt(2.0)
    t[..., 0] += 1.0
    t *= f0[:, None, :, None]
    return t


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
_engine = None


def _the_engine():
    global _engine
    if _engine is None:
        _engine = api.Engine(0)
    return _engine


def _structure(case, d):
    wfns = []
    for w in d["wfn"]:
        orbitals = [Orbital(p, e, c) for _, p, e, c in w["orbitals"]]
        wfns.append(Wavefunction(w["symbol"], w["z"], orbitals, [o for o, *_ in w["orbitals"]],
                                 list(range(len(orbitals) - 1)), [len(orbitals) - 1], w["zeta"], list(w["pow"]),
                                 w["anomalous"]))
    sg = space_group(d["group"])
    tab = case["model"] == "tab"
    types = [AtomType(np.zeros(25), 1, 1.0, 1.0, 1.0)] if tab else [
        AtomType(p, int(nl), float(v), float(k), float(kp))
        for p, nl, v, k, kp in zip(d["plm"], d["n_l"], d["p_val"], d["kappa"], d["kappa_p"])]
    n = len(d["xyz"])
    return Structure(cell=d["cell"], sg=sg, xyz=d["xyz"],
                     adp=[a[:1] if i else a for a, i in zip(d["adp"].tolist(), d["iso"])],
                     occupancy=d["occupancy"], multiplicity=np.full(n, sg.n_total, dtype=np.int32),
                     atom_wfn=d["element"].astype(np.int32),
                     atom_type=np.zeros(n, np.int32) if tab else d["type"].astype(np.int32), lcs=d["lcs"], wfns=wfns,
                     types=types, hkl=d["hkl"], dtdf=d["dtdf"], anomalous=d["anomalous"])


_PARTS = {"f": ("f",), "grad": ("f", "d_xyz", "d_adp", "d_occ"),
          "full": ("f", "d_xyz", "d_adp", "d_occ", "d_pval", "d_plm", "d_kappa", "d_kappa_prime")}
_WIDTH = {"f": 2, "d_xyz": 3, "d_adp": 6, "d_occ": 1, "d_pval": 1, "d_plm": 25, "d_kappa": 1, "d_kappa_prime": 1}


class _State:
    pass


def prepare(case, seed):
    eng = _the_engine()
    s = _State()
    s.case, s.calcs, s.crystals = case, [], _crystals(case, seed)
    s.precision = api.DSF_FP64 if case["precision"] == 64 else api.DSF_FP32_BULK
    s.options = dict(precision=s.precision, derivatives=() if case["want"] == "f" else ("xyz", "adp", "occ"),
                     multipoles=case["want"] == "full")
    for k, d in enumerate(s.crystals):
        st = _structure(case, d)
        if case["model"] == "hc":
            c = api.HcCalculator(eng, st)
        elif case["model"] == "iam":
            c = api.IamCalculator(eng, st, d["iam"])
        else:
            t = _table(d, seed, k)
            torch.cuda.synchronize()  # the engine gathers the table on its own stream
            c = api.TabulatedCalculator(eng, st, table_device=t.data_ptr())
            del t
        s.calcs.append(c)
    if case["call"] == "host":
        return s
    # device buffers: dT/dF, and one flat vector of all results (each kind over all crystals in turn)
    s.stream = torch.cuda.Stream()
    s.dtdf = [torch.tensor(d["dtdf"].view(np.float64), device="cuda") for d in s.crystals]
    parts = _PARTS[case["want"]]
    rows = lambda p, d: len(d["hkl"]) if p == "f" else len(d["xyz"])  # noqa: E731
    total = sum(_WIDTH[p] * rows(p, d) for p in parts for d in s.crystals)
    s.flat = torch.empty(total, dtype=torch.float64, device="cuda")
    s.flat32 = torch.empty(total, dtype=torch.float32, device="cuda") if case["precision"] == 32 else None
    res = s.flat if s.flat32 is None else s.flat32
    s.outputs, s.result, at = [dict() for _ in s.crystals], {}, 0
    for p in parts:
        begin = at
        for d, o in zip(s.crystals, s.outputs):
            o[p] = s.flat.data_ptr() + 8 * at
            at += _WIDTH[p] * rows(p, d)
        s.result[p] = res[begin:at].view(-1, _WIDTH[p])
    torch.cuda.synchronize()
    return s


def run(s):
    case, d = s.case, s.crystals[0]
    if case["call"] == "host":
        r = s.calcs[0].calculate(d["dtdf"], atoms=(d["xyz"], d["adp"], d["occupancy"]), adp_layout="padded",
                                 **s.options)
        if case["precision"] == 32:
            r = {k: v.astype(np.complex64 if k == "f" else np.float32) for k, v in r.items()}
        return r
    stream = s.stream.cuda_stream
    if case["count"] > 1:
        _the_engine().calculate_batch_device(s.calcs, [g.data_ptr() for g in s.dtdf], s.outputs, stream=stream,
                                             **s.options)
    else:
        if case["call"] == "cycle":
            s.calcs[0].update_types(d["plm"], d["p_val"], d["kappa"], d["kappa_p"])
            s.calcs[0].update_atoms(d["xyz"], d["adp"], d["occupancy"])
        s.calcs[0].calculate_device(s.dtdf[0].data_ptr(), s.outputs[0], stream=stream, **s.options)
    if s.flat32 is not None:
        with torch.cuda.stream(s.stream):
            s.flat32.copy_(s.flat)
    return s.result


def work(case):
    """Per term (atom x operation x reflection): the phase, the form factor, the sum and its adjoint; bytes: the
    reflections, dT/dF, atoms and (tabulated) the form factors read once, the results written once."""
    per_term = {"hc": {"f": 76, "grad": 110, "full": 195}, "iam": {"f": 30, "grad": 50, "full": 50},
                "tab": {"f": 30, "grad": 49, "full": 49}}[case["model"]][case["want"]]
    nbytes = flops = 0
    out = sum(_WIDTH[p] for p in _PARTS[case["want"]][1:])
    for n, m, g in _sizes(case):
        terms = n * m * _MULT[g]
        flops += per_term * terms
        nbytes += (8 * terms if case["model"] == "tab" else 0) + m * (12 + 16 + 16) + n * (80 + 8 * out)
        if case["model"] == "hc":
            nbytes += n * 72 + (min(case["types"], n) or n) * 28 * 8
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits, written out term by term
# ---------------------------------------------------------------------------
_NORM = [0.07957747154594767, *[0.3183098861837907] * 3, 0.75, 0.75, 0.2067483357831728, 0.75, 0.375,
         0.4244131815783876, 2.0, 0.3203330895838574, 0.2448537586029175, 0.3203330895838574, 1.0, 0.4244131815783876,
         1.875, 1.25, 0.6611826845788106, 0.4740025188689597, 0.06941752438437611, 0.4740025188689597,
         0.3305913422894053, 1.25, 0.46875]


def _harmonics(u):
    """Density-normalised real spherical harmonics to l = 4 of unit vectors [..., 3] -> [..., 25]."""
    x, y, z = u[..., 0], u[..., 1], u[..., 2]
    xx, yy, zz = x * x, y * y, z * z
    v = [torch.ones_like(x), y, z, x,
         x * y, y * z, 2 * zz - xx - yy, x * z, xx - yy,
         (3 * xx - yy) * y, x * y * z, y * (4 * zz - xx - yy), z * (2 * zz - 3 * xx - 3 * yy), x * (4 * zz - xx - yy),
         (xx - yy) * z, (xx - 3 * yy) * x,
         x * y * (xx - yy), (3 * xx - yy) * y * z, x * y * (7 * zz - 1), y * z * (7 * zz - 3),
         35 * zz * zz - 30 * zz + 3, x * z * (7 * zz - 3), (xx - yy) * (7 * zz - 1), (xx - 3 * yy) * x * z,
         xx * (xx - 3 * yy) - yy * (3 * xx - yy)]
    return torch.stack(v, -1) * torch.tensor(_NORM, dtype=u.dtype, device=u.device)


def _g(n, l, K, Z):
    """int r^n exp(-Z r) j_l(K r) dr by the recurrence over n."""
    q = Z * Z + K * K
    g0, g1 = torch.zeros_like(K), (2 * K) ** l * math.factorial(l) / q ** (l + 1)
    for i in range(l + 1, n):
        g0, g1 = g1, (2 * i * Z * g1 - (i + l) * (i - l - 1) * g0) / q
    return g1


def _g_dk(n, l, K, Z):
    return (l / K) * _g(n, l, K, Z) - _g(n + 1, l + 1, K, Z)


def _slater_pairs(orbital):
    """4 pi times the spherical density of an orbital as (coefficient, power, exponent) terms."""
    occ, po, ex, co = orbital
    return [(occ * co[i] * co[j] * (1 if i == j else 2), po[i] + po[j], ex[i] + ex[j])
            for i in range(len(co)) for j in range(i + 1)]


def _hc_radial(d, hl):
    """Per type at |h| [m]: spherical f, its parts by P_val and kappa, and the signed-free radial terms of the
    deformation density with their kappa' derivatives."""
    K = 2 * math.pi * hl
    f, fv_, dk_, r_, rk_ = [], [], [], [], []
    for t, e in enumerate(d["type_element"]):
        w = d["wfn"][int(e)]
        *core, val = w["orbitals"]
        kap, kp, pv = float(d["kappa"][t]), float(d["kappa_p"][t]), float(d["p_val"][t])
        fc = sum((c * _g(p + 2, 0, K, z) for o in core for c, p, z in _slater_pairs(o)), torch.zeros_like(K))
        terms = [(c / val[0], p, z) for c, p, z in _slater_pairs(val)]
        fv = sum(c * _g(p + 2, 0, K / kap, z) for c, p, z in terms)
        dfv = sum(c * _g_dk(p + 2, 0, K / kap, z) for c, p, z in terms) * (-K / kap ** 2)
        r, rk = [torch.zeros_like(K)] * 5, [torch.zeros_like(K)] * 5
        for l in range(min(len(w["pow"]), int(d["n_l"][t]))):
            p = w["pow"][l]
            c = 4 * math.pi * w["zeta"] ** (p + 3) / math.factorial(p + 2)
            r[l] = c * _g(p + 2, l, K / kp, w["zeta"])
            rk[l] = c * _g_dk(p + 2, l, K / kp, w["zeta"]) * (-K / kp ** 2)
        f.append(fc + pv * fv)
        fv_.append(fv)
        dk_.append(pv * dfv)
        r_.append(torch.stack(r))
        rk_.append(torch.stack(rk))
    return torch.stack(f), torch.stack(fv_), torch.stack(dk_), torch.stack(r_), torch.stack(rk_)


def _exact_one(case, d, table):
    dev, f64 = "cuda", torch.float64
    T = lambda v: torch.tensor(np.asarray(v), device=dev)  # noqa: E731
    hc, full = case["model"] == "hc", case["want"] == "full"
    ops, centro = (_SUBSET[d["group"]]) if hc else (_all_operations(d["group"]), False)
    mult = 2.0 if d["group"] == "C2/c" else 1.0
    n, m = len(d["xyz"]), len(d["hkl"])
    mm = _frac_to_cart(d["cell"])
    b = T(np.linalg.inv(mm).T)
    astar = np.linalg.norm(np.linalg.inv(mm).T, axis=0)
    lam = T(np.array([astar[i] * astar[j] for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]))
    xyz, occ, iso, adp = T(d["xyz"]), T(d["occupancy"]), T(d["iso"]), T(d["adp"])
    beta = torch.where(iso[:, None], 0.0, 2 * math.pi ** 2 * adp * lam)
    biso = torch.where(iso, 2 * math.pi ** 2 * adp[:, 0], 0.0)
    an, typ = T(d["anomalous"]), T(d["type"])
    g_in = T(d["dtdf"]).conj() * mult
    gw = (2 * g_in.real).to(torch.complex128) if centro else g_in
    if hc:
        L = T(d["lcs"])
        # crystal-frame populations: d(L^T u) = D d(u) over sample directions
        gen = torch.Generator().manual_seed(1)
        u = torch.randn((60, 3), generator=gen, dtype=f64).to(dev)
        u /= u.norm(dim=1, keepdim=True)
        v = _harmonics(u)
        D = [torch.einsum("akp,qk->apq", _harmonics(torch.einsum("aij,ki->akj", L, u))[:, :, l * l:(l + 1) ** 2],
                          torch.linalg.pinv(v[:, l * l:(l + 1) ** 2])) for l in range(5)]
        plm = T(d["plm"])[typ]
        pg = [torch.einsum("apq,ap->aq", D[l], plm[:, l * l:(l + 1) ** 2]) for l in range(5)]
    F = torch.zeros(m, dtype=torch.complex128, device=dev)
    G = {k: torch.zeros((n, w), dtype=f64, device=dev) for k, w in
         (("xyz", 3), ("six", 6), ("iso", 1), ("occ", 1), ("pv", 1), ("k", 1), ("kp", 1), ("plm", 25))}
    step = max(1, 3_000_000 // n)
    for h0 in range(0, m, step):
        hk = torch.tensor(d["hkl"][h0:h0 + step].astype(np.float64), device=dev)
        g = gw[h0:h0 + step, None]
        h2 = ((hk @ b.T) ** 2).sum(1)
        if hc:
            fs, fv, fk, r, rk = (x.index_select(0, typ) for x in _hc_radial(d, h2.sqrt()))
            r, rk = r.permute(1, 2, 0), rk.permute(1, 2, 0)
            fs = fs.T
        elif case["model"] == "iam":
            t = d["iam"]
            fs = torch.stack([float(t["c"][i]) + sum(float(t["a"][i, q]) * torch.exp(-float(t["b"][i, q]) * h2 / 4)
                                                     for q in range(4)) for i in range(len(t["c"]))]).T[:, typ]
        U = torch.zeros((len(hk), n), dtype=torch.complex128, device=dev)
        for s, (R, tr) in enumerate(ops):
            hp = hk @ torch.tensor(R, dtype=f64, device=dev)
            ph = hp @ xyz.T + (hk @ torch.tensor(tr, dtype=f64, device=dev))[:, None]
            m6 = torch.stack([hp[:, 0] ** 2, hp[:, 1] ** 2, hp[:, 2] ** 2, 2 * hp[:, 0] * hp[:, 1],
                              2 * hp[:, 0] * hp[:, 2], 2 * hp[:, 1] * hp[:, 2]], 1)
            e = torch.polar(torch.exp(-(m6 @ beta.T) - h2[:, None] * biso), 2 * math.pi * (ph - ph.round()))
            del ph
            if hc:
                y = _harmonics(hp @ b.T / h2.sqrt()[:, None])
                A = [y[:, l * l:(l + 1) ** 2] @ pg[l].T for l in range(5)]
                f = torch.complex(fs + r[0] * A[0] - r[2] * A[2] + r[4] * A[4], r[1] * A[1] - r[3] * A[3]) + an
            elif case["model"] == "iam":
                f = fs + an
            else:
                f = torch.view_as_complex(table[h0:h0 + step, s]).to(torch.complex128) + an
            u = f * e * occ
            del f
            U += u
            if case["want"] == "f":
                continue
            gu = g * u
            G["xyz"] -= 2 * math.pi * (gu.imag.T @ hp)
            G["six"] -= 2 * math.pi ** 2 * (gu.real.T @ m6) * lam
            G["iso"] -= 2 * math.pi ** 2 * (gu.real.T @ h2[:, None])
            G["occ"] += gu.real.sum(0)[:, None] / occ[:, None]
            del gu, u
            if full:
                gz = g * e * occ
                G["pv"] += (gz.real * fv.T).sum(0)[:, None]
                G["k"] += (gz.real * fk.T).sum(0)[:, None]
                for l in range(5):
                    w = (gz.real, -gz.imag, -gz.real, gz.imag, gz.real)[l]
                    G["kp"] += (w * rk[l] * A[l]).sum(0)[:, None]
                    G["plm"][:, l * l:(l + 1) ** 2] += (w * r[l]).T @ y[:, l * l:(l + 1) ** 2]
        F[h0:h0 + step] = U.sum(1)
    F = mult * (2 * F.real.to(torch.complex128) if centro else F)
    out = dict(f=torch.view_as_real(F), d_xyz=G["xyz"], d_occ=G["occ"],
               d_adp=torch.where(iso[:, None], torch.nn.functional.pad(G["iso"], (0, 5)), G["six"]))
    if full:
        out.update(d_pval=G["pv"], d_kappa=G["k"], d_kappa_prime=G["kp"])
        loc = torch.cat([torch.einsum("apq,aq->ap", D[l], G["plm"][:, l * l:(l + 1) ** 2]) for l in range(5)], 1)
        loc[:, 9:] *= T((d["n_l"] == 5).astype(np.float64))[typ][:, None]
        out["d_plm"] = loc
    return {k: out[k] for k in _PARTS[case["want"]]}


def exact(case, seed):
    if sum(n * m * _MULT[g] for n, m, g in _sizes(case)) > 2.5e10:
        return None
    got = [_exact_one(case, d, _table(d, seed, k) if case["model"] == "tab" else None)
           for k, d in enumerate(_crystals(case, seed))]
    if case["call"] == "host":
        r = {k: v.cpu().numpy() for k, v in got[0].items()}
        r["f"] = r["f"].reshape(-1).view(np.complex128)
        for k in ("d_occ", "d_pval", "d_kappa", "d_kappa_prime"):
            if k in r:
                r[k] = r[k].reshape(-1)
        if "d_kappa_prime" in r:
            r["d_kappa_p"] = r.pop("d_kappa_prime")
        return r
    return {k: torch.cat([g[k] for g in got]) for k in _PARTS[case["want"]]}

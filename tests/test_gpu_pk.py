"""pk_kernel (dsf_pk_kernel.cuh) against the CPU oracle where its tiling can go wrong: tiles of one atom, around the
32-, 64- and 128-atom marks (a small tile's warps share out the reflections), more than 32 types, reflection counts
around the sub-tile length, excluded atoms, every compiled symmetry form.

Tolerances: the plain form is held to the parity bar of the FP64 path (1e-10 relative), a factor 1e4 above the
rounding of these sums; the FP32-bulk form to its own (F 1e-6, derivatives 1e-5)."""
import numpy as np
import pytest

from conftest import rel_f, rel_norm
from discamb_gb300 import api, workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ("d_xyz", "d_adp", "d_occ")


def cut(st, n_hkl):
    idx = np.linspace(0, st.n_hkl - 1, n_hkl + 2).astype(int)[1:-1]  # not the first: an extinct axial one
    st.hkl, st.dtdf = np.ascontiguousarray(st.hkl[idx]), st.dtdf[idx]
    return st


def check(got, ref, tol, keys=KEYS, tol_f=None):
    assert rel_f(got["f"], ref["f"]) < (tol_f or tol)
    largest = max(np.linalg.norm(np.ravel(ref[k])) for k in keys)
    for k in keys:
        if np.linalg.norm(np.ravel(ref[k])) > 1e-12 * largest:
            assert rel_norm(got[k], ref[k]) < tol, k
        else:  # a class that symmetry makes zero (one extinct reflection): rounding on both sides
            assert np.linalg.norm(np.ravel(got[k])) < max(1e-12, tol * 0.1) * largest, k


def padded(ref, st):
    out = np.zeros((st.n_atoms, 6))
    for i, a in enumerate(ref["d_adp"]):
        out[i, :len(a)] = a
    return dict(ref, d_adp=out)


@pytest.mark.parametrize("n_atoms,n_hkl", [(1, 1), (2, 3), (31, 17), (33, 16), (65, 15), (70, 33), (129, 5), (200, 40)])
@pytest.mark.parametrize("sg", ["P1", "P21/c", "P212121", "P41"])
def test_fp64_tile_edges(engine, sg, n_atoms, n_hkl):
    st = cut(W.small_case(sg, n_atoms=n_atoms, stol_max=0.45, seed=900 + n_atoms), n_hkl)
    ref = padded(O.compute(st, multipoles=True), st)
    calc = api.HcCalculator(engine, st)
    keys = KEYS + ("d_pval", "d_plm", "d_kappa", "d_kappa_p")
    check(calc.calculate(st.dtdf, multipoles=True, adp_layout="padded"), ref, 1e-10, keys)
    check(calc.calculate(st.dtdf, adp_layout="padded"), ref, 1e-10)
    assert rel_f(calc.calculate(st.dtdf, derivatives=())["f"], ref["f"]) < 1e-10


@pytest.mark.parametrize("sg", ["P1", "P-1", "P21", "P21/c", "C2/c", "P212121", "Pbca", "P43212", "P3"])
def test_fp64_excluded_atoms_every_form(engine, sg):
    st = W.small_case(sg, n_atoms=37, stol_max=0.35, seed=77)
    include = np.ones(37, dtype=np.int32)
    include[::3] = 0
    st.include = include.astype(bool)
    rng = np.random.default_rng(3)
    nt = int(st.atom_type.max()) + 1
    iam = dict(ngauss=np.full(nt, 4, np.int32), a=rng.uniform(.5, 3, (nt, 5)), b=rng.uniform(.5, 30, (nt, 5)),
               c=rng.uniform(0, .5, nt))
    rots = api.all_ops_mod_centering(st.sg)[0]
    n_ops = len(rots)
    # the oracle sums the centred copies of every operation too: the same form factors for the same rotation
    every = [next(k for k in range(n_ops) if np.array_equal(rots[k], r)) for r in st.sg.rot]
    table = rng.normal(size=(st.n_hkl, n_ops, 37)) + 1j * rng.normal(size=(st.n_hkl, n_ops, 37))
    # values the widening of complex64 tables treats apart: zero, subnormal
    table[0, 0, 1], table[0, 0, 2] = 0.0, 1e-41
    for calc, ref in ((api.HcCalculator(engine, st), O.compute(st)),
                      (api.IamCalculator(engine, st, iam), O.compute(st, model="iam", iam=iam)),
                      (api.TabulatedCalculator(engine, st, table), O.compute(st, model="table", table=table[:, every])),
                      (api.TabulatedCalculator(engine, st, table, fp32_table=True),
                       O.compute(st, model="table", table=table[:, every].astype(np.complex64).astype(np.complex128)))):
        got = calc.calculate(st.dtdf, include=include, adp_layout="padded")
        check(got, padded(ref, st), 1e-10)


def test_fp64_temperature_factors_far_out(engine):
    """Displacements whose temperature factors underflow (zero there) or grow (not positive definite)."""
    st = W.small_case("P21/c", n_atoms=9, stol_max=0.5, seed=5)
    for i in range(st.n_atoms):
        a = np.array(st.adp[i])
        st.adp[i] = list(a * (4000.0 if i % 3 == 0 else -0.5 if i % 3 == 1 else 1.0))
    check(api.HcCalculator(engine, st).calculate(st.dtdf, adp_layout="padded"), padded(O.compute(st), st), 1e-10)


def shared_types(sg, n_atoms, n_types, n_hkl, seed, l_max=4):
    """A structure whose atoms share n_types types (odd and even counts: pairs with and without empty slots)."""
    st = W.small_case(sg, n_atoms=n_atoms, stol_max=0.45, seed=seed, n_types=n_types, l_max=l_max)
    return cut(st, n_hkl)


@pytest.mark.parametrize("n_atoms,n_types,n_hkl", [(1, 1, 20), (5, 5, 3), (41, 6, 17), (65, 9, 31), (127, 12, 16),
                                                   (130, 40, 15), (300, 20, 49)])
@pytest.mark.parametrize("sg", ["P1", "P21/c", "P212121", "P41", "P43212"])
def test_fp32_tile_edges(engine, sg, n_atoms, n_types, n_hkl):
    st = shared_types(sg, n_atoms, n_types, n_hkl, seed=500 + n_atoms)
    ref = padded(O.compute(st, multipoles=True), st)
    calc = api.HcCalculator(engine, st)
    keys = KEYS + ("d_pval", "d_plm", "d_kappa", "d_kappa_p")
    p = dict(precision=api.DSF_FP32_BULK, adp_layout="padded")
    check(calc.calculate(st.dtdf, multipoles=True, **p), ref, 1e-5, keys, 1e-6)
    check(calc.calculate(st.dtdf, **p), ref, 1e-5, tol_f=1e-6)
    assert rel_f(calc.calculate(st.dtdf, derivatives=(), **p)["f"], ref["f"]) < 1e-6
    check(engine.calculate_batch([calc], [st.dtdf])[0], ref, 1e-5, tol_f=1e-6)


@pytest.mark.parametrize("sg", ["P1", "P-1", "P21", "P21/c", "C2/c", "P212121", "Pbca", "P43212", "P3"])
@pytest.mark.parametrize("n_types", [6, None])
def test_fp32_excluded_atoms_every_form(engine, sg, n_types):
    st = W.small_case(sg, n_atoms=37, stol_max=0.35, seed=78, n_types=n_types)
    include = np.ones(37, dtype=np.int32)
    include[::3] = 0
    st.include = include.astype(bool)
    rng = np.random.default_rng(3)
    nt = int(st.atom_type.max()) + 1
    iam = dict(ngauss=np.full(nt, 4, np.int32), a=rng.uniform(.5, 3, (nt, 5)), b=rng.uniform(.5, 30, (nt, 5)),
               c=rng.uniform(0, .5, nt))
    for calc, ref in ((api.HcCalculator(engine, st), O.compute(st)),
                      (api.IamCalculator(engine, st, iam), O.compute(st, model="iam", iam=iam))):
        ref = padded(ref, st)
        check(calc.calculate(st.dtdf, precision=api.DSF_FP32_BULK, include=include, adp_layout="padded"), ref, 1e-5,
              tol_f=1e-6)
        check(engine.calculate_batch([calc], [st.dtdf], includes=[include])[0], ref, 1e-5, tol_f=1e-6)


@pytest.mark.parametrize("precision,tol_f,tol", [(api.DSF_FP64, 1e-10, 1e-10), (api.DSF_FP32_BULK, 1e-6, 1e-5)])
@pytest.mark.parametrize("sg", ["P21/c", "P212121", "Pbca", "P43212"])
def test_operation_order_does_not_matter(engine, sg, precision, tol_f, tol):
    """The operations in another order (the identity first) take other kernels; the sums are the same (without
    anomalous dispersion: a centrosymmetric engine combines it by the operations that it lists)."""
    from discamb_gb300.crystal import SPACE_GROUPS, SpaceGroup
    st = W.small_case(sg, n_atoms=9, stol_max=0.4, seed=12)
    for w in st.wfns:
        w.anomalous = 0j
    rng = np.random.default_rng(8)
    nt = int(st.atom_type.max()) + 1
    iam = dict(ngauss=np.full(nt, 3, np.int32), a=rng.uniform(.5, 3, (nt, 5)), b=rng.uniform(.5, 30, (nt, 5)),
               c=rng.uniform(0, .5, nt))
    ref_hc, ref_iam = padded(O.compute(st), st), padded(O.compute(st, model="iam", iam=iam), st)
    text = SPACE_GROUPS[sg]
    for order in (text[:1] + text[:0:-1], text[:1] + list(rng.permutation(text[1:]))):
        st.sg = SpaceGroup(sg, [str(v) for v in order])
        for calc, ref in ((api.HcCalculator(engine, st), ref_hc), (api.IamCalculator(engine, st, iam), ref_iam),
                          (api.HcCalculator(engine, st, representation="all"), ref_hc)):
            check(calc.calculate(st.dtdf, precision=precision, adp_layout="padded"), ref, tol, tol_f=tol_f)


def test_populations_changed_between_calls(engine):
    """update_types that empties, then fills, the l = 3, 4 populations of some types: the tiles' code follows."""
    st = shared_types("P212121", 90, 8, 60, seed=4)
    calc = api.HcCalculator(engine, st)
    full = np.array([t.plm for t in st.types])
    low = full.copy()
    low[::2, 9:] = 0.0
    for plm in (low, full):
        for t, p in zip(st.types, plm):
            t.plm = p
        calc.update_types(plm=plm)
        ref = padded(O.compute(st, multipoles=True), st)
        check(calc.calculate(st.dtdf, precision=api.DSF_FP32_BULK, multipoles=True, adp_layout="padded"), ref, 1e-5,
              KEYS + ("d_plm", "d_kappa_p"), 1e-6)
        check(calc.calculate(st.dtdf, precision=api.DSF_FP32_BULK, adp_layout="padded"), ref, 1e-5, tol_f=1e-6)
        check(calc.calculate(st.dtdf, adp_layout="padded"), ref, 1e-10)


def device_call(calc, st, multipoles):
    """A call on device buffers as a function of its settings, its stream and its output buffers."""
    import torch

    n, stream = st.n_atoms, torch.cuda.Stream()
    dev = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")
    out = {"f": dev(2 * st.n_hkl), "d_xyz": dev(3 * n), "d_adp": dev(6 * n), "d_occ": dev(n)}
    if multipoles:
        out.update(d_pval=dev(n), d_plm=dev(25 * n), d_kappa=dev(n), d_kappa_prime=dev(n))
    g = torch.from_numpy(np.ascontiguousarray(st.dtdf).view(np.float64).ravel().copy()).cuda()
    torch.cuda.synchronize()

    def call(precision, multipoles=multipoles):
        calc.calculate_device(g.data_ptr(), {k: v.data_ptr() for k, v in out.items()}, precision=precision,
                              multipoles=multipoles, stream=stream.cuda_stream)

    return call, stream, out


def check_device(out, st, precision):
    """Output buffers of a device call against the oracle."""
    got = {k: v.cpu().numpy() for k, v in out.items()}
    got["f"] = got["f"].view(np.complex128)
    if "d_kappa_prime" in got:
        got["d_kappa_p"] = got.pop("d_kappa_prime")
    ref = padded(O.compute(st, multipoles="d_pval" in got), st)
    tol, tol_f = (1e-10, 1e-10) if precision == api.DSF_FP64 else (1e-5, 1e-6)
    check({k: v.reshape(np.shape(ref[k])) for k, v in got.items()}, ref, tol, [k for k in got if k != "f"], tol_f)


def scale_kappa(calc, st, factor):
    kappa = np.array([factor * t.kappa for t in st.types])
    for t, k in zip(st.types, kappa):
        t.kappa = k
    calc.update_types(kappa=kappa)


@pytest.mark.parametrize("precision", [api.DSF_FP32_BULK, api.DSF_FP64])
@pytest.mark.parametrize("multipoles", [False, True])
def test_first_call_under_capture(engine, precision, multipoles):
    """The first call after update_types is a captured one: it builds the tables that it reads."""
    import torch

    st = shared_types("P21", 40, 8, 50, seed=6)
    calc = api.HcCalculator(engine, st)
    call, stream, out = device_call(calc, st, multipoles)
    scale_kappa(calc, st, 1.04)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call(precision)
    graph.replay()
    torch.cuda.synchronize()
    check_device(out, st, precision)


def test_populations_changed_under_a_captured_call(engine):
    """A captured FP32 call replayed after update_types reads the new radial tables (kappa moves
    them all), also where no other call came between."""
    import torch

    st = shared_types("P21", 40, 8, 50, seed=6)
    calc = api.HcCalculator(engine, st)
    n, stream = st.n_atoms, torch.cuda.Stream()
    dev = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")
    out = {"f": dev(2 * st.n_hkl), "d_xyz": dev(3 * n), "d_adp": dev(6 * n), "d_occ": dev(n)}
    g = torch.from_numpy(np.ascontiguousarray(st.dtdf).view(np.float64).ravel().copy()).cuda()

    def call():
        calc.calculate_device(g.data_ptr(), {k: v.data_ptr() for k, v in out.items()},
                              precision=api.DSF_FP32_BULK, stream=stream.cuda_stream)

    torch.cuda.synchronize()
    call()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    kappa = np.array([1.04 * t.kappa for t in st.types])
    for t, k in zip(st.types, kappa):
        t.kappa = k
    calc.update_types(kappa=kappa)
    graph.replay()
    torch.cuda.synchronize()
    ref = padded(O.compute(st), st)
    got = {k: v.cpu().numpy() for k, v in out.items()}
    got["f"] = got["f"].view(np.complex128)
    check({k: v.reshape(np.shape(ref[k])) for k, v in got.items()}, ref, 1e-5, tol_f=1e-6)


@pytest.mark.parametrize("precision", [api.DSF_FP32_BULK, api.DSF_FP64])
@pytest.mark.parametrize("entry", ["single", "batch"])
def test_every_captured_call_follows_the_types(engine, precision, entry):
    """A captured call with the multipole adjoint reads the new tables after update_types, radial terms and kappa
    derivatives alike, also where the last call before asked for less."""
    import torch

    st = shared_types("P21", 40, 8, 50, seed=6)
    calc = api.HcCalculator(engine, st)
    call, stream, out = device_call(calc, st, True)
    if entry == "batch":
        g = torch.from_numpy(np.ascontiguousarray(st.dtdf).view(np.float64).ravel().copy()).cuda()
        torch.cuda.synchronize()

        def call(precision, multipoles=True):
            engine.calculate_batch_device([calc], [g.data_ptr()], [{k: v.data_ptr() for k, v in out.items()}],
                                          precision=precision, multipoles=multipoles, stream=stream.cuda_stream)
    call(precision)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call(precision)
    call(precision, False)
    stream.synchronize()
    scale_kappa(calc, st, 1.04)
    graph.replay()
    torch.cuda.synchronize()
    check_device(out, st, precision)


def random_iam(st, seed, terms=4):
    rng = np.random.default_rng(seed)
    nt = int(st.atom_type.max()) + 1
    return dict(ngauss=np.full(nt, terms, np.int32), a=rng.uniform(.5, 3, (nt, 5)), b=rng.uniform(.5, 30, (nt, 5)),
                c=rng.uniform(0, .5, nt))


@pytest.mark.parametrize("sg", ["P1", "P-1", "P21", "P21/c", "C2/c", "P212121", "Pbca", "P43212", "P3"])
@pytest.mark.parametrize("n_atoms", [5, 37, 130])
def test_independent_atoms_structure_factors_only(engine, sg, n_atoms):
    """derivatives=(): the forward-only kernels of the FP32 independent-atom model, and the FP64 call."""
    st = W.small_case(sg, n_atoms=n_atoms, stol_max=0.35, seed=78, n_types=6)
    iam = random_iam(st, 3)
    calc = api.IamCalculator(engine, st, iam)
    ref = O.compute(st, model="iam", iam=iam)["f"]
    for precision, tol in ((api.DSF_FP32_BULK, 1e-6), (api.DSF_FP64, 1e-10)):
        assert rel_f(calc.calculate(st.dtdf, precision=precision, derivatives=())["f"], ref) < tol


def test_more_tiles_than_a_grid_dimension_holds(engine):
    """65,537 tiles: copies of a 128-atom cell with occupancies of their own.  F is the small cell's times the sum of
    the factors, an atom's derivatives the small cell's (by position and ADP times its factor)."""
    copies = 65537
    st = W.small_case("P1", n_atoms=128, stol_max=0.35, seed=31, n_types=5)
    st.adp = np.random.default_rng(2).uniform(0.02, 0.05, (128, 6)) * np.array([1, 1, 1, .2, .2, .2])
    st = cut(st, 3)
    iam = random_iam(st, 3)
    ref = O.compute(st, model="iam", iam=iam)
    factor = np.random.default_rng(4).uniform(0.5, 1.5, copies)
    big = W.small_case("P1", n_atoms=128, stol_max=0.35, seed=31, n_types=5)
    big.hkl, big.dtdf = st.hkl, st.dtdf
    big.xyz, big.adp = np.tile(st.xyz, (copies, 1)), np.tile(st.adp, (copies, 1))
    big.occupancy = np.outer(factor, st.occupancy).ravel()
    for k in ("multiplicity", "atom_wfn", "atom_type"):
        setattr(big, k, np.tile(getattr(st, k), copies))
    if st.anomalous is not None:
        big.anomalous = np.tile(st.anomalous, copies)
    calc = api.IamCalculator(engine, big, iam)
    want = {"d_xyz": np.multiply.outer(factor, ref["d_xyz"]).reshape(-1, 3),
            "d_adp": np.multiply.outer(factor, np.array(ref["d_adp"])).reshape(-1, 6), "d_occ": np.tile(ref["d_occ"], copies)}
    for precision, tol in ((api.DSF_FP64, 1e-10), (api.DSF_FP32_BULK, 1e-5)):
        got = calc.calculate(big.dtdf, precision=precision, adp_layout="padded")
        assert rel_f(got["f"], ref["f"] * factor.sum()) < min(tol, 1e-6)
        for k, v in want.items():
            assert rel_norm(got[k], v) < tol, k
            # no tile left out: the largest difference of any atom
            assert np.abs(got[k] - v).max() < 10 * tol * np.abs(v).max(), k
    calc.close()


def test_two_threads_with_different_shared_memory(engine):
    """Two host threads launch one kernel with 5 and with 32 types per tile (other shared-memory sizes) at once: FP64
    batches, which launch per structure."""
    import threading

    import torch

    failed, jobs = [], []
    for n_types in (5, 60):
        st = shared_types("P1", 120, n_types, 16, seed=8)
        calcs = [api.HcCalculator(engine, st) for _ in range(16)]
        parts = [device_call(c, st, True) for c in calcs]
        g = torch.from_numpy(np.ascontiguousarray(st.dtdf).view(np.float64).ravel().copy()).cuda()
        jobs.append((st, calcs, [p[2] for p in parts], g, parts[0][1]))
    torch.cuda.synchronize()

    def many(st, calcs, outs, g, stream):
        try:
            for _ in range(200):
                engine.calculate_batch_device(calcs, [g.data_ptr()] * len(calcs),
                                              [{k: v.data_ptr() for k, v in o.items()} for o in outs],
                                              precision=api.DSF_FP64, multipoles=True, stream=stream.cuda_stream)
        except api.DsfError as exc:
            failed.append(exc)

    threads = [threading.Thread(target=many, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed
    for st, _, outs, _, _ in jobs:
        for out in outs:
            check_device(out, st, api.DSF_FP64)


# operation lists in the usual order, beside those of crystal.SPACE_GROUPS
LISTS = {
    "P4/m": "x,y,z;-x,-y,z;-y,x,z;y,-x,z;-x,-y,-z;x,y,-z;y,-x,-z;-y,x,-z",
    "P422, 222 first": "x,y,z;-x,-y,z;x,-y,-z;-x,y,-z;-y,x,z;y,-x,z;y,x,-z;-y,-x,-z",
}
HC, BOTH = ("hc",), ("hc", "iam", "table")


@pytest.mark.parametrize("sg,models", [("P1", BOTH), ("P-1", BOTH), ("P21", BOTH), ("P21/c", BOTH), ("C2/c", BOTH),
                                       ("P212121", BOTH), ("Pbca", BOTH), ("P41", HC), ("P43212", BOTH),
                                       ("P422, 222 first", BOTH), ("P4/m", BOTH), ("P3", ()), ("Fdd2", ())])
def test_which_kernel_a_listed_group_takes(engine, sg, models):
    """Every group whose operations have a compiled form takes pk_kernel (its records' kind), the others the general
    kernel, and FP32 tables always that."""
    from discamb_gb300.crystal import SpaceGroup
    st = W.small_case("P43212" if sg in LISTS else sg, n_atoms=12, stol_max=0.3, seed=3, n_types=5)
    if sg in LISTS:
        st.sg = SpaceGroup(sg, LISTS[sg].split(";"))
    ops = len(api.all_ops_mod_centering(st.sg)[0])
    calcs = {"hc": api.HcCalculator(engine, st), "iam": api.IamCalculator(engine, st, random_iam(st, 3)),
             "table": api.TabulatedCalculator(engine, st, np.ones((st.n_hkl, ops, 12), complex))}
    for model, calc in calcs.items():
        kinds = [calc.debug_kernel_kind(api.DSF_FP32_BULK), calc.debug_kernel_kind(api.DSF_FP32_BULK, multipoles=True),
                 calc.debug_kernel_kind(api.DSF_FP64)]
        want = [-1, -1, -1] if model not in models else {"hc": [0, 1, 2], "iam": [0, 0, 2], "table": [-1, -1, 2]}[model]
        assert kinds == want, model


@pytest.mark.parametrize("sg", list(LISTS))
def test_eight_operations_without_compiled_cosets(engine, sg):
    """Generic models with eight operations in no compiled coset form, against the oracle."""
    from discamb_gb300.crystal import SpaceGroup
    st = W.small_case("P43212", n_atoms=37, stol_max=0.35, seed=77)
    st.sg = SpaceGroup(sg, LISTS[sg].split(";"))
    iam = random_iam(st, 3)
    rng = np.random.default_rng(3)
    table = rng.normal(size=(st.n_hkl, 8, 37)) + 1j * rng.normal(size=(st.n_hkl, 8, 37))
    for calc, ref in ((api.IamCalculator(engine, st, iam), O.compute(st, model="iam", iam=iam)),
                      (api.TabulatedCalculator(engine, st, table), O.compute(st, model="table", table=table))):
        ref = padded(ref, st)
        check(calc.calculate(st.dtdf, adp_layout="padded"), ref, 1e-10)
        check(calc.calculate(st.dtdf, precision=api.DSF_FP32_BULK, adp_layout="padded"), ref, 1e-5, tol_f=1e-6)
        check(engine.calculate_batch([calc], [st.dtdf])[0], ref, 1e-5, tol_f=1e-6)


def many_blocks(sg, n_types):
    """8,000 atoms of both ADP kinds and 10,240 reflections in whole lattice lines: 63 and more tiles in chunks of 256
    reflections are over 16 blocks per SM, where FP32 calls take one launch per ADP kind."""
    cell = (64.0, 64.0, 72.0, 90.0, 90.0, 90.0)
    laue = {"P1": 2, "P-1": 2, "P21": 4, "P21/c": 4, "P41": 8, "P212121": 8, "Pbca": 8, "P43212": 16}[sg]
    rng = np.random.default_rng(60)
    # reflections to s: 4/3 pi (2 s)^3 V, one in `laue` of them unique, and a third more
    stol = (1.35 * 10240 * laue / (32 * np.pi / 3 * 64 * 64 * 72)) ** (1 / 3)
    st = W.build_structure(cell=cell, sg_symbol=sg, elements=W.protein_elements(8000, rng), rng=rng, n_types=n_types,
                           stol_max=stol)
    order = np.lexsort(st.hkl.T[::-1])[:10240]
    st.hkl, st.dtdf = np.ascontiguousarray(st.hkl[order]), st.dtdf[order]
    assert st.n_hkl == 10240 and len(set(map(len, st.adp))) == 2
    return st


def against_fp64(calc, st, **kw):
    a = calc.calculate(st.dtdf, precision=api.DSF_FP64, adp_layout="padded", **kw)
    b = calc.calculate(st.dtdf, precision=api.DSF_FP32_BULK, adp_layout="padded", **kw)
    assert rel_f(b["f"], a["f"]) < 1e-6
    for k in a:
        if k != "f" and kw.get("derivatives") != ():
            assert rel_norm(b[k], a[k]) < 1e-5, k


@pytest.mark.parametrize("sg", ["P1", "P-1", "P21", "P21/c", "P41", "P212121", "Pbca", "P43212"])
def test_fp32_one_launch_per_adp_kind(engine, sg):
    """Calls large enough for a launch per ADP kind, with straight groups of reflections, against the FP64 call."""
    st = many_blocks(sg, 60)
    calc = api.HcCalculator(engine, st)
    assert calc.debug_kernel_kind(api.DSF_FP32_BULK) == 0
    against_fp64(calc, st)
    against_fp64(calc, st, multipoles=True)
    against_fp64(calc, st, derivatives=())
    calc.close()
    calc = api.IamCalculator(engine, st, random_iam(st, 3))
    against_fp64(calc, st)
    against_fp64(calc, st, derivatives=())
    calc.close()


@pytest.mark.parametrize("sg", ["P1", "P-1", "P212121", "P43212"])
def test_fp32_one_launch_per_adp_kind_a_type_per_atom(engine, sg):
    """The same with types of one or two atoms: one atom per thread."""
    st = many_blocks(sg, 6000)
    calc = api.HcCalculator(engine, st)
    assert calc.debug_kernel_kind(api.DSF_FP32_BULK) == 1
    against_fp64(calc, st)
    against_fp64(calc, st, multipoles=True)
    against_fp64(calc, st, derivatives=())
    calc.close()


@pytest.mark.parametrize("n_hkl,kind", [(1000, -1), (10240, 0)])
def test_isotropic_independent_atoms_with_eight_operations(engine, n_hkl, kind):
    """Isotropic structures with eight operations in no coset form take the general kernel when they are small; both
    sides of the rule against the FP64 call."""
    st = many_blocks("P43212", 60)
    st.adp = [a[:1] for a in st.adp]
    st = st.subset(np.arange(900))
    st.hkl, st.dtdf = st.hkl[:n_hkl], st.dtdf[:n_hkl]
    iam = random_iam(st, 3)
    calc = api.IamCalculator(engine, st, iam)
    assert calc.debug_kernel_kind(api.DSF_FP32_BULK) == kind
    against_fp64(calc, st)
    against_fp64(calc, st, derivatives=())
    a = calc.calculate(st.dtdf, adp_layout="padded")
    check(engine.calculate_batch([calc], [st.dtdf])[0], a, 1e-5, tol_f=1e-6)
    calc.close()

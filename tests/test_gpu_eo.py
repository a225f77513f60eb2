"""GPU even-odd (site parity) family against the oracle (on the CASE0, 4 and 7
lattices) and the CASE0 golden.

main.cc fills its arrays with the DD generator and reads them with the
even-odd operators too; oracle/qwsref.py's eo_perm gives the field an
even-odd operator sees, eo_partner the aliasing of half-array arguments.
Tolerances: FP64 1e-13, FP32 1e-6 (relative norm of the difference).
"""
import json
from pathlib import Path

import numpy as np
import pytest

from qwsref import Oracle, check_sh_ok, eo_partner, eo_perm, gen_main_fields, parity_mask

pytestmark = pytest.mark.gpu

GOLD = json.loads((Path(__file__).parent / "golden" / "case_norms.json").read_text())
KAPPA = 0.05
FAC = -KAPPA * KAPPA
# (pe, which, dag, clov, mode) of the reference's entry points
COMBOS = [(1, 1, 0, 0, 0), (1, 1, 0, 1, 0), (1, 1, 1, 0, 0), (1, 1, 1, 1, 0), (1, 1, 0, 1, 2),
          (1, 1, 1, 0, 2), (1, 2, 0, 0, 1), (1, 2, 1, 0, 1), (1, 2, 0, 1, 1), (1, 2, 1, 1, 1),
          (1, 3, 0, 0, 0), (1, 3, 0, 1, 0), (1, 3, 1, 0, 0), (1, 3, 1, 1, 0), (1, 3, 0, 1, 2),
          (1, 3, 1, 0, 2), (0, 3, 0, 1, 2)]


def rel(a, b, m):
    a, b = np.asarray(a, np.float64)[m], np.asarray(b, np.float64)[m]
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


# golden lattices whose global extents are all even (site parity is then
# consistent across the periodic boundaries)
EO_CASES = {
    "CASE0": ((32, 6, 4, 3), (1, 1, 1, 1)),
    "CASE4": ((32, 6, 6, 2), (1, 1, 1, 2)),
    "CASE7": ((32, 6, 4, 3), (1, 2, 2, 2)),
}


@pytest.fixture(scope="module", params=list(EO_CASES))
def setup(request):
    import qws_b200

    lloc, npe = EO_CASES[request.param]
    L = tuple(a * b for a, b in zip(lloc, npe))
    NB = (2 * npe[0], npe[1], npe[2], npe[3])
    U, C, S = gen_main_fields(lloc, npe, 2)
    if request.param == "CASE0":  # the even-odd reading of main.cc's arrays
        P = eo_perm(L)
        U, C, b = U[:, P], C[P], S[0][P]
    else:
        b = S[0]
    o = Oracle(L, NB, tbc=-1, kappa=KAPPA)
    o.set_fields(U, C)
    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=KAPPA)
    lat.load_fields(U, C)
    yield request.param, L, o, lat, b
    lat.close()


@pytest.mark.parametrize("combo", COMBOS)
def test_deo_combos(setup, combo):
    name, L, o, lat, b = setup
    pe, which, dag, clov, mode = combo
    m = parity_mask(L, pe)
    in0 = b[eo_partner(L)]
    acc0 = np.random.default_rng(7).standard_normal(b.shape)
    for dt, tol in ((np.float64, 1e-13), (np.float32, 1e-6)):
        x, i0, a0 = b.astype(dt), in0.astype(dt), acc0.astype(dt)
        ref = o.deo(x, pe, which, dag, clov, mode, dt(FAC), i0 if mode == 2 else None,
                    out=a0.copy() if mode == 1 else None)
        got = lat.to_host(lat.deo(lat.to_device(x), pe, which, dag, clov, mode, FAC,
                                  in0=lat.to_device(i0) if mode == 2 else None,
                                  out=lat.to_device(a0) if mode == 1 else None))
        assert rel(got, ref, m) < tol, (dt, combo)


def test_mtilde_and_solver(setup):
    name, L, o, lat, b = setup
    m0 = parity_mask(L, 0)
    xd = lat.to_device(b)
    assert rel(lat.to_host(lat.mtilde(xd)), o.mtilde(b), m0) < 1e-13
    assert rel(lat.to_host(lat.mtilde(xd, dag=True)), o.mtilde(b, True), m0) < 1e-13
    be = b * m0[:, None]
    xo, it_o = o.bicgstab_vm(be, np.zeros_like(b), 100)
    x = lat.empty("f64")
    it = lat.bicgstab_vm(x, lat.to_device(be), 100)
    assert abs(it - it_o) <= 1
    assert rel(lat.to_host(x), xo, m0) < 1e-11
    if name == "CASE0":
        assert it == 91  # the golden's timing table: 91 bicgstab_iter_ calls
        r = be - o.mtilde(lat.to_host(x))
        n2 = lambda a: float(np.sum(a[m0] ** 2))
        vals = [v for k, v in GOLD["CASE0"]["norms"] if k in ("bnorm^2", "rnorm^2", "xnorm^2")][:3]
        for nm_, val, ref in zip(("bnorm^2", "rnorm^2", "xnorm^2"),
                                 (n2(be), n2(r), n2(lat.to_host(x))), vals):
            assert check_sh_ok(nm_, val, ref), (nm_, val, ref)


def test_cg_solvers(setup):
    """cg_vm_ (cg.cc:65) and mcg_vm_ (mcg.cc:65) on mtilde^dag mtilde against
    the oracle's restatements (which tests/test_oracle_vs_ref.py pins to the
    reference's own solvers): iteration counts within 2% (about a thousand
    iterations on an ill-conditioned operator, where the sums' rounding moves
    the count by a few), solutions to 1e-10 relative (both stop at
    |r|/|b| < 1e-14; the condition number is ~4e3), and every shifted
    system solved to 1e-10."""
    name, L, o, lat, b = setup
    m0 = parity_mask(L, 0)
    be = b * m0[:, None]
    bd = lat.to_device(be)
    xo, it_o = o.cg_vm(be, np.zeros_like(b), 3000)
    assert it_o < 2999
    x = lat.empty("f64")
    it = lat.cg_vm(x, bd, 3000)
    assert abs(it - it_o) <= max(1, it_o // 50)
    assert rel(lat.to_host(x), xo, m0) < 1e-10
    sigma = [0.0, 0.05, 0.5, 2.0]
    Xo, it_o = o.mcg_vm(be, sigma, 3000)
    X, it = lat.mcg_vm(bd, sigma, 3000)
    assert abs(it - it_o) <= max(1, it_o // 50)
    for k, s in enumerate(sigma):
        xk = lat.to_host(X[k])
        assert np.isfinite(xk).all(), k
        assert rel(xk, Xo[k], m0) < 1e-10, k
        ax = lat.to_host(lat.mtdagmt(X[k])) + s * xk
        assert rel(ax, be, m0) < 1e-10, k


@pytest.mark.parametrize("L, NB", [((6, 5, 3, 2), (2, 1, 1, 2)), ((10, 6, 14, 4), (2, 2, 2, 2)),
                                   ((4, 2, 2, 4), (2, 1, 1, 1))])
def test_compact_layout_at_edges(L, NB):
    """Extents 2 and 3, odd extents and parities that do not fill a block: the
    Schur operators against the oracle, FP64 1e-13 and FP32 1e-6, the other
    parity of the output untouched."""
    import qws_b200

    U, _ = qws_b200.gen_gauge(L, 3, 2, 0.36)
    C = qws_b200.gen_clover(U, L, 1.0, 0.12)
    b = qws_b200.gen_source(L, 4)
    o = Oracle(L, NB, tbc=-1, kappa=0.12)
    o.set_fields(U, C)
    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.12)
    lat.load_fields(U, C)
    try:
        m0 = parity_mask(L, 0)
        fill = np.full_like(b, 7.0)
        for dag in (False, True):
            got = lat.to_host(lat.mtilde(lat.to_device(b), dag=dag, out=lat.to_device(fill)))
            assert rel(got, o.mtilde(b, dag), m0) < 1e-13
            assert np.array_equal(got[~m0], fill[~m0])
        bs = b.astype(np.float32)
        assert rel(lat.to_host(lat.mtilde(lat.to_device(bs))), o.mtilde(b), m0) < 1e-6
    finally:
        lat.close()


def test_compact_fields_follow_changes():
    """The compact copies are made again after every change of the fields, on
    the handle itself and on a one-RHS handle that borrows them."""
    import qws_b200

    L, NB = (8, 4, 4, 6), (2, 1, 1, 1)
    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.12)
    try:
        x = lat.to_device(qws_b200.gen_source(L, 4))
        child = None
        for seed in (3, 5):
            lat.gen_gauge_device(seed, 2, 0.36)
            for csw in (1.0, 1.5):
                lat.build_clover(csw)
                child = child or lat.batch(1)
                fresh = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.12)
                fresh.gen_gauge_device(seed, 2, 0.36)
                fresh.build_clover(csw)
                want = fresh.to_host(fresh.mtilde(x))
                fresh.close()
                assert np.array_equal(lat.to_host(lat.mtilde(x)), want)
                assert np.array_equal(child.to_host(child.mtilde(x)), want)
    finally:
        if child:
            child.close()
        lat.close()


def fresh_lattice(L, NB, seed, csw=1.0, stream=None):
    import qws_b200

    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.12, stream=stream)
    lat.gen_gauge_device(seed, 2, 0.36)
    lat.build_clover(csw)
    return lat


def device_memory_of(f):
    """bytes of device memory that f() took and kept (after a first run of
    the same kernels elsewhere, which loads them)"""
    import torch

    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    f()
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0]


def test_deo_takes_no_memory():
    """One hop operator reads and writes the full planes: no copy of the
    fields and no work vector, also on the handle's first call."""
    import torch

    L, NB = (16, 16, 16, 16), (2, 1, 1, 1)
    taken = []
    for _ in range(2):  # (the first handle loads the kernels)
        lat = fresh_lattice(L, NB, 3)
        x = {dt: lat.to_device(np.ones((lat.V, 24), dt)) for dt in (np.float64, np.float32)}
        out = {dt: torch.zeros_like(v) for dt, v in x.items()}
        taken.append(device_memory_of(lambda: [lat.deo(x[dt], 1, clov=1, out=out[dt]) for dt in x]))
        lat.close()
    assert taken[1] == 0


def test_captured_deo_on_a_fresh_handle():
    """The first call on a handle inside a stream capture; the replay reads the
    fields as they are then."""
    import qws_b200
    import torch

    L, NB = (8, 4, 4, 6), (2, 1, 1, 1)
    st = torch.cuda.Stream()
    lat = fresh_lattice(L, NB, 3, stream=st)
    x = lat.to_device(qws_b200.gen_source(L, 4))
    out = torch.zeros_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        lat.deo(x, 1, clov=1, out=out)
    for seed in (3, 5):
        lat.gen_gauge_device(seed, 2, 0.36)
        lat.build_clover(1.5)
        g.replay()
        torch.cuda.synchronize()
        want = fresh_lattice(L, NB, seed, 1.5)
        assert torch.equal(out, want.deo(x, 1, clov=1))
        want.close()
    lat.close()


@pytest.mark.parametrize("L, NB", [((6, 5, 3, 2), (2, 1, 1, 1)), ((10, 6, 14, 4), (2, 2, 2, 2)),
                                   ((10, 3, 3, 3), (2, 1, 1, 1)), ((4, 2, 2, 4), (2, 1, 1, 1))])
@pytest.mark.parametrize("combo", [(0, 3, 0, 1, 0), (1, 1, 1, 0, 2), (0, 2, 0, 1, 1), (1, 3, 0, 0, 1)])
def test_deo_at_edges(L, NB, combo):
    """Rows of odd length (a pair of neighbouring sites of one parity, or none
    of it), extents 2 and 3: FP64 1e-13 and FP32 1e-6 against the oracle, the
    other parity of the output untouched."""
    import qws_b200

    U, _ = qws_b200.gen_gauge(L, 3, 2, 0.36)
    C = qws_b200.gen_clover(U, L, 1.0, 0.12)
    b, in0, acc0 = (qws_b200.gen_source(L, 4 + k) for k in range(3))
    o = Oracle(L, NB, tbc=-1, kappa=0.12)
    o.set_fields(U, C)
    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.12)
    lat.load_fields(U, C)
    pe, which, dag, clov, mode = combo
    m = parity_mask(L, pe)
    try:
        for dt, tol in ((np.float64, 1e-13), (np.float32, 1e-6)):
            x, i0, a0 = b.astype(dt), in0.astype(dt), acc0.astype(dt)
            ref = o.deo(x, pe, which, dag, clov, mode, dt(FAC), i0 if mode == 2 else None,
                        out=a0.copy())
            got = lat.to_host(lat.deo(lat.to_device(x), pe, which, dag, clov, mode, FAC,
                                      in0=lat.to_device(i0) if mode == 2 else None,
                                      out=lat.to_device(a0)))
            assert rel(got, ref, m) < tol, (dt, combo)
            assert np.array_equal(got[~m], a0[~m])
    finally:
        lat.close()


def schur_ops(lat, b):
    """{name: (operator, input, output)} of the Schur operators"""
    import torch

    x = lat.to_device(b)
    xs = lat.to_device(b.astype(np.float32))
    ops = {"mtilde": lambda x, o: lat.mtilde(x, out=o),
           "mtilde_dag": lambda x, o: lat.mtilde(x, dag=True, out=o),
           "mtdagmt": lambda x, o: lat.mtdagmt(x, out=o)}
    ops = {k: (f, x, torch.zeros_like(x)) for k, f in ops.items()}
    ops["mtilde_s"] = (lambda x, o: lat.mtilde(x, out=o), xs, torch.zeros_like(xs))
    return ops


def close(a, b):
    """two FP64 (FP32) results of the same sums, 8 hops and two 6x6 products
    deep: 1e-14 (1e-6) relative"""
    tol = 1e-14 if a.element_size() == 8 else 1e-6
    return float((a - b).norm() / b.norm()) < tol


@pytest.mark.parametrize("L, NB", [((8, 4, 4, 6), (2, 1, 1, 1)), ((10, 6, 14, 4), (2, 2, 2, 2))])
def test_captured_schur_operators_follow_fields(L, NB):
    """A graph captured after one call replays on the fields as they are then,
    and a capture leaves nothing behind that the next plain call would take for
    made."""
    import qws_b200
    import torch

    st = torch.cuda.Stream()
    b = qws_b200.gen_source(L, 4)
    lat = fresh_lattice(L, NB, 3, stream=st)
    ops = schur_ops(lat, b)
    ops["mtilde"][0](*ops["mtilde"][1:])  # the first use makes the work vectors
    torch.cuda.synchronize()
    graphs = {}
    for name, (f, x, out) in ops.items():
        graphs[name] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[name], stream=st):
            f(x, out)
    for seed in (5, 7):
        lat.gen_gauge_device(seed, 2, 0.36)
        lat.build_clover(1.5)
        want = fresh_lattice(L, NB, seed, 1.5)
        for name, (f, x, out) in schur_ops(want, b).items():
            f(x, out)
            torch.cuda.synchronize()
            graphs[name].replay()
            torch.cuda.synchronize()
            assert close(ops[name][2], out), (seed, name)
        if seed == 5:  # captured after a change of the fields, before any plain call on them
            g = torch.cuda.CUDAGraph()
            f, x, out = ops["mtdagmt"]
            with torch.cuda.graph(g, stream=st):
                f(x, out)
        for name, (f, x, out) in schur_ops(want, b).items():  # plain calls
            f(x, out)
            ops[name][0](*ops[name][1:])
            torch.cuda.synchronize()
            assert torch.equal(ops[name][2], out), (seed, name)
        want.close()
    lat.close()


@pytest.mark.parametrize("bytes_a_site", [1450, 2000])
def test_without_room_for_a_copy_of_the_fields(bytes_a_site):
    """With that many bytes of device memory a site left, all operators and solvers
    run, to the same results: 1,450 hold the work vectors (480 bytes a site of
    the operators', 576 more of the solvers') but no copy of the fields (1,152
    in FP64) beside them; 2,000 hold a copy until the solvers need their
    vectors.  Once there is room again they use a copy."""
    import qws_b200
    import torch

    L, NB = (16, 16, 16, 32), (2, 1, 1, 1)
    b = qws_b200.gen_source(L, 4)
    solvers = {"bicgstab": lambda l, x, d: l.bicgstab_vm(x, d, 200),
               "cg": lambda l, x, d: l.cg_vm(x, d, 1000)}
    runs = []
    for scarce in (False, True):  # (the first handle loads the kernels)
        lat = fresh_lattice(L, NB, 3)
        ops, bd = schur_ops(lat, b), lat.to_device(b)
        xs = {name: torch.zeros_like(bd) for name in solvers}
        runs.append((ops, xs))
        if not scarce:  # the kernels on full planes
            lat.deo(bd, 0, clov=1)
            for dag in (0, 1):
                for mode, clov in ((0, 1), (2, 1 - dag)):
                    lat.deo(bd, 0, dag=dag, clov=clov, mode=mode, in0=bd)
                    lat.deo(bd.float(), 0, dag=dag, clov=clov, mode=mode, in0=bd.float())
            lat.clv(bd, 0)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill, chunk, keep = [], 2 << 20, bytes_a_site * lat.V
        while scarce and (free := torch.cuda.mem_get_info()[0]) > keep + chunk:
            fill.append(torch.empty((free - keep) // chunk * chunk, dtype=torch.uint8, device="cuda"))
        try:
            for f, x, out in ops.values():
                f(x, out)
            for name, f in solvers.items():
                f(lat, xs[name], bd)
            torch.cuda.synchronize()
        finally:
            fill.clear()
            torch.cuda.empty_cache()
        if scarce:
            for name in solvers:
                assert float((xs[name] - runs[0][1][name]).norm() / xs[name].norm()) < 1e-11, name
            for again in (False, True):
                for name, (f, x, out) in ops.items():
                    want = runs[0][0][name][2]
                    assert torch.equal(out, want) if again else close(out, want), (name, again)
                    f(x, out)
                torch.cuda.synchronize()
        lat.close()


def test_borrowing_handles_share_the_copy_of_the_fields():
    """A one-RHS handle reads its lattice's copy of the fields: its first call
    takes its work vectors (480 bytes a site and the allocations' rounding),
    not a copy (1,152) of its own."""
    L, NB = (16, 16, 16, 32), (2, 1, 1, 1)
    taken = []
    for _ in range(2):  # (the first pair loads the kernels)
        lat = fresh_lattice(L, NB, 3)
        x = lat.to_device(np.ones((lat.V, 24)))
        want = lat.mtdagmt(x)
        child = lat.batch(1)
        out = child.empty("f64")
        taken.append(device_memory_of(lambda: child.mtdagmt(x, out=out)))
        assert np.array_equal(lat.to_host(out), lat.to_host(want))
        child.close()
        lat.close()
    assert taken[1] < 600 * 16 ** 3 * 32 + (4 << 20)


def test_threads_share_the_copy_of_the_fields():
    """A lattice and two handles on its fields, a thread and a stream each, make
    their first calls after a change of the fields at the same time."""
    import threading

    import qws_b200
    import torch

    L, NB = (12, 8, 6, 10), (2, 2, 1, 1)
    b = qws_b200.gen_source(L, 4)
    lat = fresh_lattice(L, NB, 1)
    handles = [lat, lat.batch(1), lat.batch(1)]
    for h in handles:
        h.use_own_stream()
    x, outs = lat.to_device(b), [h.empty("f64") for h in handles]
    for seed in range(1, 9):
        lat.gen_gauge_device(seed, 2, 0.36)
        lat.build_clover(1.0)
        torch.cuda.synchronize()
        start = threading.Barrier(len(handles))

        def work(h, out):
            start.wait()
            for _ in range(3):
                h.mtdagmt(x, out=out)

        ts = [threading.Thread(target=work, args=a) for a in zip(handles, outs)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        torch.cuda.synchronize()
        want = fresh_lattice(L, NB, seed)
        w = want.mtdagmt(x)
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o in outs), seed
        want.close()
    for h in handles[1:] + [lat]:
        h.close()


def test_shift_vectors_are_given_back():
    """mcg_vm's vectors: an outgrown block goes back, and a call for which there
    is no room takes nothing."""
    import qws_b200
    import torch

    L, NB = (16, 16, 16, 16), (2, 1, 1, 1)
    lat = fresh_lattice(L, NB, 3)
    X = torch.zeros(32 * 24 * lat.pad, dtype=torch.float64, device="cuda")
    bd = lat.to_device(qws_b200.gen_source(L, 4))

    def mcg(n):  # two iterations, into X
        import ctypes

        sigma, it = np.linspace(0.0, 1.0, n), ctypes.c_int()
        return lat.lib.qwsg_mcg_vm(lat.h, X.data_ptr(), bd.data_ptr(), n,
                                   ctypes.c_void_p(sigma.ctypes.data), 3, ctypes.byref(it))

    one_shift = 2 * 96 * lat.V
    assert mcg(2) == 0
    grown = device_memory_of(lambda: [mcg(n) for n in (3, 4, 6, 8)])
    assert grown < 6 * one_shift + (4 << 20)
    torch.cuda.empty_cache()
    fill, chunk, keep = [], 2 << 20, 14 * one_shift
    while (free := torch.cuda.mem_get_info()[0]) > keep + chunk:
        fill.append(torch.empty((free - keep) // chunk * chunk, dtype=torch.uint8, device="cuda"))
    try:
        # 32 shifts do not fit, not even with the block of eight and the copy of
        # the fields (6 shifts' worth) given back for them
        rc = []
        taken = device_memory_of(lambda: rc.extend(mcg(32) for _ in range(3)))
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    assert 0 not in rc and taken < 0
    assert mcg(32) == 0
    lat.close()


def test_copies_give_way_to_other_work_buffers():
    """After an even-odd operator, with 1,400 bytes of device memory a site left,
    a DD solve whose buffers need 2,208 takes those of the copy of the fields
    (1,152), and the operator still runs."""
    import qws_b200
    import torch

    L, NB = (16, 16, 16, 32), (2, 1, 1, 1)
    res = []
    for scarce in (False, True):  # (the first handle loads the kernels)
        lat = fresh_lattice(L, NB, 3)
        bd = lat.to_device(qws_b200.gen_source(L, 4))
        x, out, again = (torch.zeros_like(bd) for _ in range(3))
        lat.mtdagmt(bd, out=out)
        lat.deo(bd, 0, clov=1, out=again)
        lat.ddd(bd, out=again)
        lat.ddd(bd.float())
        again.zero_()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill, chunk, keep = [], 2 << 20, 1400 * lat.V
        while scarce and (free := torch.cuda.mem_get_info()[0]) > keep + chunk:
            fill.append(torch.empty((free - keep) // chunk * chunk, dtype=torch.uint8, device="cuda"))
        try:
            lat.bicgstab_dd_mix(x, bd, 1e-10, 20, 1e-6, 50)
            lat.mtdagmt(bd, out=again)
            torch.cuda.synchronize()
        finally:
            fill.clear()
            torch.cuda.empty_cache()
        assert close(again, out)
        res.append(x)
        lat.close()
    assert torch.equal(*res)

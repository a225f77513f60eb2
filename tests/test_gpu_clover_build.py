"""Fields built on the GPU against the host generators that follow the same
conventions: the clover term (qwsg_build_clover vs qwsg_gen_clover) and the
seeded smoothed gauge field (qwsg_gen_gauge_device vs qwsg_gen_gauge).  The
FP64 operator with either field agrees to 1e-13 / 1e-12, the FP32 one to
FP32 rounding, and a solve gives the same iterations.  The free field
(U = 1, F = 0) must give the trivial clover term 1/2 on the diagonal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = (8, 8, 8, 16)
KAPPA, CSW = 0.1365, 1.7


def rel(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("NB", [(2, 1, 1, 1), (2, 2, 2, 2)])
def test_device_clover_matches_host(NB):
    import qws_b200

    U, _ = qws_b200.gen_gauge(L, 5, 5, 0.36)
    C = qws_b200.gen_clover(U, L, CSW, KAPPA)
    b = qws_b200.gen_source(L, 9)
    host = qws_b200.Lattice(L, NB, tbc=-1, kappa=KAPPA)
    dev = qws_b200.Lattice(L, NB, tbc=-1, kappa=KAPPA)
    try:
        host.load_fields(U, C)
        dev.load_gauge(U)
        dev.build_clover(CSW)
        for dt, tol in ((np.float64, 1e-13), (np.float32, 1e-6)):
            x = b.astype(dt)
            assert rel(dev.to_host(dev.ddd(dev.to_device(x))),
                       host.to_host(host.ddd(host.to_device(x)))) < tol, dt
        xs = [lat.empty("f64") for lat in (host, dev)]
        st = [lat.bicgstab_dd_mix(x, lat.to_device(b), 1e-10, 100, 1e-6, 50)
              for lat, x in zip((host, dev), xs)]
        assert abs(st[0]["outer_iters"] - st[1]["outer_iters"]) <= 1
        assert rel(dev.to_host(xs[1]), host.to_host(xs[0])) < 1e-8
    finally:
        host.close()
        dev.close()


def test_free_field_clover_is_trivial():
    import qws_b200

    V = int(np.prod(L))
    U = np.zeros((4, V, 3, 3, 2))
    for c in range(3):
        U[:, :, c, c, 0] = 1.0
    lat = qws_b200.Lattice(L, (2, 2, 2, 2), tbc=-1, kappa=KAPPA)
    ref = qws_b200.Lattice(L, (2, 2, 2, 2), tbc=-1, kappa=KAPPA)
    try:
        lat.load_gauge(U)
        lat.build_clover(CSW)
        C = np.zeros((V, 72))
        C[:, 0:6] = 0.5
        C[:, 36:42] = 0.5
        ref.load_fields(U, C)
        b = qws_b200.gen_source(L, 3)
        got = lat.to_host(lat.ddd(lat.to_device(b)))
        want = ref.to_host(ref.ddd(ref.to_device(b)))
        assert rel(got, want) < 1e-15
    finally:
        lat.close()
        ref.close()


def test_device_gauge_matches_host():
    """qwsg_gen_gauge_device draws the same random streams and applies the same
    smoothing as the host generator: the operators built on the two fields
    agree to rounding, and so do the plaquettes."""
    import qws_b200

    U, plaq = qws_b200.gen_gauge(L, 21, 5, 0.36)
    host = qws_b200.Lattice(L, (2, 2, 2, 2), tbc=-1, kappa=KAPPA)
    dev = qws_b200.Lattice(L, (2, 2, 2, 2), tbc=-1, kappa=KAPPA)
    try:
        host.load_gauge(U)
        p = dev.gen_gauge_device(21, 5, 0.36)
        assert abs(p - plaq) < 1e-12, (p, plaq)
        host.build_clover(CSW)
        dev.build_clover(CSW)
        b = qws_b200.gen_source(L, 4)
        assert rel(dev.to_host(dev.ddd(dev.to_device(b))),
                   host.to_host(host.ddd(host.to_device(b)))) < 1e-12
    finally:
        host.close()
        dev.close()


@pytest.mark.parametrize("shape, NB, csw", [
    ((6, 3, 5, 2), (2, 1, 1, 2), 1.7),      # odd extents, extent 2, a ragged last block
    ((18, 18, 22, 20), (2, 2, 2, 2), 1.7),  # walks of 4 sites, extents not multiples of 4
    ((4, 4, 6, 8), (2, 1, 1, 1), 12.0),     # indefinite blocks: the pivoted inverse
])
def test_clover_operator_at_edges(shape, NB, csw):
    """A^-1 on every site, FP64: A^-1 v of the device-built term against the
    host generator's.  Both are backward-stable inverses of the same T, so
    they differ by its condition number (below 1e3 but for rare sites of the
    indefinite case) in FP64 roundoffs."""
    import qws_b200

    U, _ = qws_b200.gen_gauge(shape, 8, 5, 0.36)
    C = qws_b200.gen_clover(U, shape, csw, KAPPA)
    host = qws_b200.Lattice(shape, NB, tbc=-1, kappa=KAPPA)
    dev = qws_b200.Lattice(shape, NB, tbc=-1, kappa=KAPPA)
    try:
        host.load_fields(U, C)
        dev.load_gauge(U)
        dev.build_clover(csw)
        x = qws_b200.gen_source(shape, 9)
        for p in (0, 1):
            got = dev.to_host(dev.clv(dev.to_device(x), p))
            want = host.to_host(host.clv(host.to_device(x), p))
            assert rel(got, want) < (1e-13 if csw < 2 else 1e-10), p
    finally:
        host.close()
        dev.close()


def test_batch_with_some_indefinite_blocks():
    """A kappa per right-hand side, of which one gives indefinite clover blocks
    (the pivoted inverse, at that right-hand side's entries alone): the FP64 and
    FP32 operators and the FP16 SAP of every right-hand side against those of a
    lattice with that kappa.  Both sides make the same clover term, bit for bit,
    and run the same sums, so FP64 and FP32 differ by at most a rounding of the
    result (2^-53, 2^-24 relative) and the SAP by that of its FP16 storage in
    each of its sweeps (2^-11, four times)."""
    import qws_b200

    shape, NB, csw = (4, 4, 6, 8), (2, 1, 1, 1), 12.0
    kappas = [0.002, KAPPA, 0.001, 0.003]
    U, _ = qws_b200.gen_gauge(shape, 8, 5, 0.36)
    lat = qws_b200.Lattice(shape, NB, tbc=-1, kappa=0.002)
    many = None
    try:
        lat.load_gauge(U)
        lat.build_clover(csw)
        many = lat.batch(4)
        many.set_kappas(kappas, csw)
        x = np.stack([qws_b200.gen_source(shape, 9 + r) for r in range(4)])
        xd, xs = many.to_device(x), many.to_device(x.astype(np.float32))
        got = {"ddd": many.to_host(many.ddd(xd)), "ddd_s": many.to_host(many.ddd(xs)),
               "prec_h": many.to_host(many.prec_h(xs, 2, 2))}
        for r, k in enumerate(kappas):
            lat.set_kappa(k)
            lat.build_clover(csw)
            one, ones = lat.to_device(x[r]), lat.to_device(x[r].astype(np.float32))
            assert rel(got["ddd"][r], lat.to_host(lat.ddd(one))) < 2**-53, k
            assert rel(got["ddd_s"][r], lat.to_host(lat.ddd(ones))) < 2**-24, k
            assert rel(got["prec_h"][r], lat.to_host(lat.prec_h(ones, 2, 2))) < 4 * 2**-11, k
    finally:
        if many:
            many.close()
        lat.close()

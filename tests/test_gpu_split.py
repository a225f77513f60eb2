"""The four-threads-a-site kernels of small launches against the one-thread
kernels, which a handle with two right-hand sides runs: FP32 results equal bit
for bit, on site counts that leave the last CTA of 32 sites partly filled,
with 12-real and full links, and on both sides of the size at which launches
change over (FP16 21,312 and FP32 31,968 sites a launch)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L, NB, links12", [
    ((6, 6, 2, 10), (2, 1, 1, 2), True),      # 360 sites a colour, odd block extents
    ((12, 6, 6, 6), (2, 2, 2, 2), False),     # one-site interiors, full links
    ((4, 4, 4, 4), (4, 2, 2, 2), True),       # blocks one site wide along x
    ((16, 12, 14, 16), (2, 2, 2, 2), True),   # 21,504 a colour: FP32 below, FP16 above
])
def test_split_kernels_equal_one_thread_kernels(L, NB, links12):
    import qws_b200

    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.13)
    two = None
    try:
        lat.set_link_compression(1 if links12 else 0)
        lat.gen_gauge_device(5, 2, 0.36)
        lat.build_clover(1.2)
        two = lat.batch(2)
        v = [qws_b200.gen_source(L, 20 + k).astype(np.float32) for k in range(2)]
        b1, b2 = lat.to_device(v[0]), two.to_device(np.stack(v))
        ops = {"ddd": lambda h, b: h.ddd(b), "prec": lambda h, b: h.prec(b, 3, 2),
               "prec_ddd": lambda h, b: h.prec_ddd(b, 3, 2), "prec_h": lambda h, b: h.prec_h(b, 3, 2)}
        for c in (0, 1):
            ops["in%d" % c] = lambda h, b, c=c: h.ddd_in(b, c)
            ops["out%d" % c] = lambda h, b, c=c: h.ddd_out(b, c, 0.7, out=b.clone())
            ops["out_h%d" % c] = lambda h, b, c=c: h.ddd_out_h(b, c, 0.7, out=b.clone())
            ops["jinv%d" % c] = lambda h, b, c=c: h.jinv(b, c, 3)
            ops["jinv_h%d" % c] = lambda h, b, c=c: h.jinv_h(b, c, 3)
        for name, f in ops.items():
            assert np.array_equal(lat.to_host(f(lat, b1)), two.to_host(f(two, b2))[0]), name
    finally:
        if two:
            two.close()
        lat.close()

"""The algorithmic bytes behind the SAP update's reported bandwidth: each
spinor, link and clover term a launch needs, once, counted site by site."""
import itertools
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def update_bytes(L, NB, links12):
    """FP32 bytes of one update of colour 0 with all hops: s (read and
    written), in, a, links and clover of its sites, and of the other colour the
    spins of a that its hops read and the links of its backward hops"""
    B = [l // n for l, n in zip(L, NB)]
    colour = lambda x: sum(c // b for c, b in zip(x, B)) % 2
    spins, links, sites = {}, set(), 0
    for x in itertools.product(*map(range, L)):
        if colour(x) != 0:
            continue
        sites += 1
        for mu in range(4):
            for d in (1, -1):
                y = list(x)
                y[mu] = (y[mu] + d) % L[mu]
                y = tuple(y)
                if colour(y) == 0:
                    continue
                # a hop in t reads two of the four spins, by direction
                half = {1 if d > 0 else 2} if mu == 3 else {1, 2}
                spins[y] = spins.get(y, set()) | half
                if d < 0:
                    links.add((y, mu))
    link = 48 if links12 else 72
    return (sites * (4 * 96 + 4 * link + 288) + sum(48 * len(s) for s in spins.values())
            + len(links) * link)


@pytest.mark.parametrize("L, NB", [((8, 6, 4, 8), (2, 1, 1, 1)), ((8, 6, 4, 8), (2, 2, 2, 2)),
                                   ((12, 4, 2, 6), (4, 2, 1, 2)), ((8, 4, 4, 2), (2, 1, 1, 2))])
@pytest.mark.parametrize("links12", [True, False])
def test_sap_update_bytes(L, NB, links12):
    import qws_b200

    lat = qws_b200.Lattice(L, NB, tbc=-1, kappa=0.12)
    try:
        lat.set_link_compression(1 if links12 else 0)
        lat.gen_gauge_device(5, 1, 0.36)
        lat.build_clover(1.0)
        b = lat.to_device(np.ones((math.prod(L), 24), np.float32))
        lat.prec_ddd(b, 2, 2)  # (every update of it has all hops)
        lat.kernel_timing(True)
        lat.prec_ddd(b, 2, 2)
        n, _, nbytes = lat.kernel_stats()["sap_update_f32"]
        assert n == 4
        assert nbytes / n == pytest.approx(update_bytes(L, NB, links12), rel=1e-12)
    finally:
        lat.close()

"""Periodic halos: one launch whose tiles cover 32 rows (x), 32 points of the 8 halo rows
(y) and 32 x 8 points of a halo plane (z).  Every haloed point of every face against the
wrapped interior, at sizes that cut the tiles, for a box and for a grid with one periodic
direction; copies, so the same bits.
"""
import numpy as np
import pytest

from ocfd_testlib import curvilinear_case, tgv_case
from ocfd_b200.solver import Solver

pytestmark = pytest.mark.gpu

L = 4  # halo layers


@pytest.mark.parametrize("n", [(8, 8, 9), (33, 17, 10), (65, 40, 9), (16, 33, 70)], ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("box", [True, False], ids=["box", "span"])
def test_face_halos(box, n, mixed):
    if not box:  # the boundary closures need more points than the smallest box
        n = (max(n[0], 16), max(n[1], 16), n[2])
    p, mesh, prims = tgv_case(n=n, mixed=mixed) if box else curvilinear_case(n=n)
    p.precision = 1 if mixed else 0
    rng = np.random.default_rng(9)
    prims = [a * (1.0 + 1e-2 * rng.normal(size=a.shape)) for a in prims]
    s = Solver(p)
    s.init_mesh(*(mesh or ()))
    s.init3d(prims)
    s.exchange_boundary_xyz()
    got = s.download_state()[1]
    s.close()
    for q in range(5):
        g = got[q]
        core = g[L:-L, L:-L, L:-L]
        for axis, per in ((2, box), (1, box), (0, True)):
            if not per:
                continue
            pad = [(L, L) if a == axis else (0, 0) for a in range(3)]
            want = np.pad(core, pad, mode="wrap")
            have = g[tuple(slice(None) if a == axis else slice(L, -L) for a in range(3))]
            np.testing.assert_array_equal(have, want)

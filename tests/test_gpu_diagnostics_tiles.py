"""Diagnostics whose blocks walk runs of 256 points of a plane (Q in rows of 64 and more:
tiles of 32 x 8): planes smaller than a run, runs and tiles cut in
each direction, more tiles than blocks, box and body-fitted grids.  Q and the time
averages are point by point (the strict build gives the oracle's bits); the sums of
show_flow_msg and ana_box are taken in another order: n eps bounds the difference of two
orders for terms of one sign (n = 150,000 at most: 3.4e-11), 1e-10 as for the small case
elsewhere where ana_box divides by small moments.
"""
import numpy as np
import pytest

from ocfd_testlib import curvilinear_case, rel_err, tgv_case
from ocfd_b200.solver import Solver
from pyoracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strict", [True, False], ids=["strict", "fast"])
@pytest.mark.parametrize("n", [(8, 8, 9), (33, 9, 10), (31, 23, 8), (64, 40, 57), (8, 37, 60), (13, 35, 40)], ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("box", [True, False], ids=["box", "curvilinear"])
def test_diagnostics(box, n, strict):
    if not box:  # the boundary closures need more points than the smallest box
        n = (max(n[0], 16), max(n[1], 16), n[2])
    p, mesh, prims = tgv_case(n=n) if box else curvilinear_case(n=n)
    rng = np.random.default_rng(5)
    prims = [a * (1.0 + 1e-2 * rng.normal(size=a.shape)) for a in prims]
    o, s = Oracle(p), Solver(p, strict=strict)
    for x in (o, s):
        x.init_mesh(*(mesh or ()))
        x.init3d(prims)
        x.step(1)
    mean = np.zeros((5, p.nz, p.ny, p.nx))
    s.ana_time_average()
    o.ana_time_average(mean, 0)
    q, avg = s.ana_q(), np.stack(s.download_average()[0])
    if strict:
        np.testing.assert_array_equal(q, o.ana_q())
        np.testing.assert_array_equal(avg, mean)
    else:
        assert rel_err(q, o.ana_q()) < 1e-10
        assert rel_err(avg, mean) < 1e-12
    assert rel_err(s.show_flow_msg(), o.show_flow_msg()) < 1e-10
    assert rel_err(s.ana_box()[1:], o.ana_box()[1:]) < 1e-10
    s.close()
    o.close()

"""Small grids run the three sweeps and the viscous gradients of a stage in one launch.
The stage operators launch them one by one: the same bits, for every scheme and form, at
sizes with tiles cut in each direction, rows with and without a 16-byte stride.  The
launches of a step tell which it was: 64x31x65 is just below the limit of 1 MiB an array in
FP64, 64x32x65 just above it (in mixed precision both are far below).
"""
import numpy as np
import pytest

from ocfd_testlib import tgv_case
from ocfd_b200.params import (SCHEME_HYBRID, SCHEME_OMP6, SCHEME_UD7L, SCHEME_WENO5, SCHEME_WENO7, SPLIT_LLF,
                              SPLIT_SW)
from ocfd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [(24, 20, 16), (33, 17, 8), (65, 9, 33), (64, 31, 65), (64, 32, 65)], ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("scheme,character,split", [
    (SCHEME_WENO5, 0, SPLIT_LLF), (SCHEME_WENO7, 0, SPLIT_SW), (SCHEME_OMP6, 0, SPLIT_SW), (SCHEME_UD7L, 0, SPLIT_SW),
    (SCHEME_HYBRID, 0, SPLIT_LLF), (SCHEME_WENO5, 1, SPLIT_SW), (SCHEME_WENO7, 1, SPLIT_SW), (SCHEME_OMP6, 1, SPLIT_SW),
    (SCHEME_UD7L, 1, SPLIT_LLF), (SCHEME_HYBRID, 1, SPLIT_SW)])
def test_one_launch_equals_four(scheme, character, split, n, mixed):
    p, mesh, prims = tgv_case(scheme=scheme, character=character, split=split, n=n, ma=0.5, mixed=mixed)
    rng = np.random.default_rng(11)
    prims = [a * (1.0 + 5e-3 * rng.normal(size=a.shape)) for a in prims]
    a, b = Solver(p), Solver(p)
    for s in (a, b):
        s.init_mesh(*(mesh or ()))
        s.init3d(prims)
    a.stage_step()
    b.step(1)
    # three stages of sweeps and gradients, tail, repair; the sensor and its halos once a step
    merged = mixed or n != (64, 32, 65)
    assert b.step_kernels() == 3 * (3 if merged else 6) + (2 if scheme == SCHEME_HYBRID else 0)
    fa, fb = a.download_f(), b.download_f()
    a.close()
    b.close()
    np.testing.assert_array_equal(fa, fb)

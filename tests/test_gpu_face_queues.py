"""Face sweeps whose uncommon faces leave the common path: the hybrid scheme's WENO
faces, the OMP6 limiter, the boundary closures of the characteristic form.

A noisy field makes every kind of face occur in one tile; the sizes put the ends of
pencils and planes at, before and past the tile edges (16, 32 and 64 faces, 8 and 16
pencils).  An odd nx has rows of no 16-byte stride, so its tiles are staged with plain
loads, an even one's by TMA.  du of one stage against the oracle within 1e-10 of
max|du|, the production build's bar in test_gpu_parity.py (du is a difference of face
fluxes about 200 times larger, so a few ulp of them show as 1e-13).

Mixed precision: the same du, from the same FP64 state (so the sensor and the class of
every face are the oracle's), within K eps32 S; S is the largest energy flux (|u| + c)(E + p)
over the smallest distance of two points, the size of a face flux in du.  K = 20: du takes
six faces, each with some 16 roundings of half an eps (inputs, splitting, scheme), 48 eps
if all were of one sign; the largest seen is 14.4.
"""
import numpy as np
import pytest

from ocfd_testlib import curvilinear_case, rel_err, tgv_case
from ocfd_b200.params import SCHEME_HYBRID, SCHEME_OMP6, SCHEME_WENO5, SCHEME_WENO7, SPLIT_LLF, SPLIT_SW
from ocfd_b200.solver import Solver
from pyoracle import Oracle

pytestmark = pytest.mark.gpu

BOX = [(24, 20, 16), (33, 17, 8), (64, 9, 32), (65, 16, 33)]
WALLS = [(25, 21, 8), (24, 20, 8), (65, 18, 9)]


def _noisy(prims, amp):
    rng = np.random.default_rng(7)
    return [a * (1.0 + amp * rng.normal(size=a.shape)) + (0.01 * rng.normal(size=a.shape) if q == 3 else 0.0)
            for q, a in enumerate(prims)]


K = 20.0


def _flux_scale(p, mesh, prims):
    d, u, v, w, T = prims
    pr = d * T / (p.gamma * p.ma ** 2)
    q2 = u * u + v * v + w * w
    e = (np.sqrt(q2) + np.sqrt(T) / p.ma) * (p.gamma / (p.gamma - 1.0) * pr + 0.5 * d * q2)
    if mesh is None:
        h = 2.0 * np.pi / max(p.nx, p.ny, p.nz)
    else:
        h = min(np.sqrt(sum(np.diff(x, axis=a) ** 2 for x in mesh)).min() for a in range(3))
    return float(e.max() / h)


def _compare(p, mesh, prims, mixed=False):
    if p.scheme_invis == SCHEME_HYBRID:
        p.hybrid_para[0], p.hybrid_para[1], p.hybrid_para[2], p.hybrid_para[3] = 1, 0.004, 0.01, 0
        p.ud7l_diss = 0.3
    pm = p.copy()
    pm.precision = 1 if mixed else 0
    o, s = Oracle(p), Solver(pm)
    for x in (o, s):
        x.init_mesh(*(mesh or ()))
        x.init3d(prims)
    o.halo_prims()
    s.exchange_boundary_xyz()
    if p.scheme_invis == SCHEME_HYBRID:
        o.comput_rhybrid()
        s.comput_Rhybrid()
    if p.if_scheme_character:
        o.du_inviscous_character()
        s.du_inviscous_Character()
    else:
        o.du_inviscous()
        s.du_inviscous()
    du, ref = s.download_du(), np.array(o.du)
    s.close()
    o.close()
    if mixed:
        err = float(np.abs(du - ref).max()) / (np.finfo(np.float32).eps * _flux_scale(p, mesh, prims))
        assert err <= K, err
    else:
        err = rel_err(du, ref)
        assert err <= 1e-10, err


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed32"])
@pytest.mark.parametrize("n", BOX, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("amp", [2e-3, 2e-2], ids=["mixed", "rough"])
@pytest.mark.parametrize("scheme,character,split", [
    (SCHEME_HYBRID, 0, SPLIT_LLF), (SCHEME_HYBRID, 1, SPLIT_SW), (SCHEME_OMP6, 1, SPLIT_SW), (SCHEME_WENO7, 0, SPLIT_SW),
    (SCHEME_WENO7, 1, SPLIT_LLF), (SCHEME_WENO5, 0, SPLIT_LLF), (SCHEME_HYBRID, 0, SPLIT_SW), (SCHEME_HYBRID, 1, SPLIT_LLF)])
def test_periodic_sweeps(scheme, character, split, amp, n, mixed):
    p, mesh, prims = tgv_case(scheme=scheme, character=character, split=split, n=n, ma=0.5)
    _compare(p, mesh, _noisy(prims, amp), mixed)


@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed32"])
@pytest.mark.parametrize("n", WALLS, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("ghost", [True, False], ids=["ghost", "oneside"])
@pytest.mark.parametrize("scheme", [SCHEME_WENO5, SCHEME_WENO7, SCHEME_OMP6, SCHEME_HYBRID])
def test_boundary_closures(scheme, ghost, n, mixed):
    p, mesh, prims = curvilinear_case(scheme=scheme, n=n, ghost=ghost)
    _compare(p, mesh, _noisy(prims, 5e-3), mixed)

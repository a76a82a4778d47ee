"""Mixed-precision runs of the hybrid scheme keep their bits.

The hybrid's sensor is a hard threshold on the state: a last-bit change of an FP32 face
flux moves faces beside a front between the linear scheme and WENO, and two roundings of
the same flux part by far more than they differ.  So the FP32 arithmetic of these sweeps
is fixed, and the fields of short runs are pinned to it, bit for bit: both splittings,
both forms, grids below and above the size of the merged stage launch, rows with and
without a 16-byte stride, a batch, and a body-fitted grid with walls (general metric
row, boundary closures).  All inputs are made without transcendental functions, so that
they are the same on every host.  The digests belong to nvcc 12.9 (the compiler
contracts the sums of these sweeps).
"""
import hashlib

import numpy as np
import pytest

from ocfd_b200 import cases
from ocfd_b200.params import SCHEME_HYBRID, SPLIT_LLF, SPLIT_SW
from ocfd_b200.solver import Batch, Solver

pytestmark = pytest.mark.gpu

BOX = {"small": (24, 20, 16), "odd": (33, 17, 9), "large": (72, 64, 60)}
FORMS = {"flux-llf": (0, SPLIT_LLF), "flux-sw": (0, SPLIT_SW), "char-sw": (1, SPLIT_SW), "char-llf": (1, SPLIT_LLF)}

DIGESTS = {
    "flux-llf-small": "a4b22d18dc36b8cc",
    "flux-llf-odd": "1857cc3bfb011d1c",
    "flux-llf-large": "5da583566dbe96f5",
    "flux-sw-small": "55be8ab2654e2e7d",
    "flux-sw-odd": "460a89d6aad56d9f",
    "flux-sw-large": "76a9c8428f677e67",
    "char-sw-small": "030375be9a8b5ed1",
    "char-sw-odd": "5ce07c96f94a7e0c",
    "char-sw-large": "da0ce6c31cddc470",
    "char-llf-small": "6b38e04226f98dc5",
    "char-llf-odd": "7a08efe01958ba4d",
    "char-llf-large": "7027f1b72e6fb49e",
    "flux-llf-wall40": "ae018a1067e185f5",
    "flux-llf-wall41": "1c6234fd8decbcb1",
    "flux-sw-wall40": "a1fc720473745eed",
    "flux-sw-wall41": "bf73aa7a0e3ff0f2",
    "char-sw-wall40": "d1d501a4aad02349",
    "char-sw-wall41": "eaf7ddd3299d48b7",
    "char-llf-wall40": "f9d571e194c5229f",
    "char-llf-wall41": "47fec170e8e85898",
    "batch": "a4b22d18dc36b8cc+1857cc3bfb011d1c",
}


def _bump(n):
    """A periodic bump in [0, 1], polynomial on each half."""
    x = (np.arange(n) + 0.5) / n
    return 16.0 * (x * (1.0 - x)) ** 2


def _prims(n):
    """Smooth flow, a steep patch and small noise: faces of the three classes in every sweep."""
    nx, ny, nz = n
    rng = np.random.default_rng(29)
    x, y, z = _bump(nx)[None, None, :], _bump(ny)[None, :, None], _bump(nz)[:, None, None]
    patch = np.zeros((nz, ny, nx))
    patch[nz // 4:nz // 2, ny // 4:ny // 2, nx // 4:nx // 2] = 1.0
    noise = [2e-3 * (rng.random((nz, ny, nx)) - 0.5) for _ in range(5)]
    d = 1.0 + 0.05 * x * y + 0.3 * patch
    T = 1.0 + 0.05 * y * z + 0.1 * patch
    u, v, w = 0.5 * y + 0.1 * z - 0.3, 0.4 * z * x - 0.2, 0.5 * x + 0.1 * y - 0.2
    return [np.ascontiguousarray(np.broadcast_to(a, d.shape) * (1.0 + e)) + (e if q in (1, 2, 3) else 0.0)
            for q, (a, e) in enumerate(zip((d, u, v, w, T), noise))]


def _params(p, form):
    p.scheme_invis = SCHEME_HYBRID
    p.if_scheme_character, p.flux_splitting = FORMS[form]
    p.hybrid_para[0], p.hybrid_para[1], p.hybrid_para[2], p.hybrid_para[3] = 1, 0.02, 0.1, 0
    p.ud7l_diss = 0.125
    p.precision = 1
    return p


def _box(form, n):
    s = Solver(_params(cases.tgv_params(n[0], ny=n[1], nz=n[2], ma=0.5, dt=0.01), form))
    s.init_mesh()
    s.init3d(_prims(n))
    return s


def _wall(form, n, ghost):
    ni, nj, nk = n
    p = _params(cases.cylinder_params(ni, nj, nk, ma=3.0, re=1e4, dt=2e-4), form)
    if not ghost:
        p.ghost_cell[2] = 0
        p.scheme_boundary[2] = 0
    # a curved channel: stretched towards j = 1, both families of lines curved
    a, b = np.arange(ni)[None, :] / (ni - 1.0), np.arange(nj)[:, None] / (nj - 1.0)
    X2 = a + 0.1 * b * (1.0 - b) * (2.0 * a - 1.0)
    Y2 = 0.7 * b * (0.4 + 0.6 * b) + 0.2 * a * (1.0 - a) * (1.0 - b)
    z = 0.1 * np.arange(nk) / nk
    shape = (nk, nj, ni)
    s = Solver(p)
    s.init_mesh(*(np.broadcast_to(q, shape).copy() for q in (X2, Y2, z[:, None, None])))
    s.init3d(_prims(n))
    return s


def _digest(s):
    return hashlib.sha256(np.ascontiguousarray(s.download_f()).tobytes()).hexdigest()[:16]


def _runs():
    """name -> function that returns the digest."""
    def one(make, *args):
        s = make(*args)
        s.step(4)
        r = _digest(s)
        s.close()
        return r

    def batch():
        ss = [_box("flux-llf", BOX["small"]), _box("flux-llf", BOX["odd"])]
        b = Batch(ss)
        b.step(4)
        r = "+".join(_digest(s) for s in ss)
        b.close()
        for s in ss:
            s.close()
        return r

    out = {f"{form}-{size}": (one, _box, form, n) for form in FORMS for size, n in BOX.items()}
    for form in FORMS:
        for n in ((40, 33, 8), (41, 32, 9)):
            out[f"{form}-wall{n[0]}"] = (one, _wall, form, n, n[0] == 40)
    out["batch"] = (batch,)
    return out


@pytest.mark.parametrize("name", list(_runs()))
def test_bits_of_mixed_hybrid_runs(name):
    f, *args = _runs()[name]
    assert f(*args) == DIGESTS[name]

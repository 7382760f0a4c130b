"""The reversed face kernels of the adjoint over the schemes, limiters, fluids and models they
branch on, each against central differences of the GPU residual (the checks and the
tolerance of test_gpu_adjoint), and the adjoint through a mixed-form engine."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, adjoint, native
from tests import test_gpu_adjoint as base

pytestmark = pytest.mark.gpu

# nscheme, nmuscl, nlim, fluid, iturb
VARIANTS = [(1, 2, 8, 2, 0), (2, 2, 8, 2, 0), (3, 2, 8, 2, 0), (4, 0, 0, 2, 0), (4, 1, 1, 2, 0), (1, 2, 3, 2, -2),
            (4, 2, 2, 2, -2), (4, 2, 4, 2, -3), (4, 2, 5, 2, 0), (1, 2, 6, 2, -3), (4, 2, 7, 2, 0),
            (1, 1, 8, 1, 0), (4, 2, 8, 1, -2)]


def _case(nscheme, nmuscl, nlim, fluid, iturb):
    c = base._state(8)
    c["cfg"].update(nscheme=nscheme, nmuscl=nmuscl, nlim=nlim, fluid=fluid, iturb=iturb)
    if fluid == 1:
        c["cfg"].update(ncav=0)
    npv = abi.sizes(c["cfg"])[0]
    c["pv0"] = [np.ascontiguousarray(c["pv0"][0][..., :npv])]
    return c


@pytest.mark.parametrize("variant", VARIANTS, ids=lambda v: "-".join(map(str, v)))
def test_vjp_variants(variant):
    c = _case(*variant)
    e = native.Engine(c, precision=abi.FP64)
    e.initialize(c["pv0"])
    s = adjoint.StateSetter(e)
    pv = s.interior(0)
    res = s.residual([pv])[0]
    rng = np.random.default_rng(5)
    scale = np.abs(res).reshape(-1, res.shape[-1]).max(axis=0)
    lam = rng.normal(size=res.shape) / np.maximum(scale, 1e-300)
    g, _ = e.residual_vjp([lam])
    d = dict(pv=pv, lam=lam, g=g[0])
    entries = base._entries(pv.shape[:-1], pv.shape[-1], 18, 7)
    used, errs, rows = base._check(lambda p: s.residual([p])[0], d, entries)
    assert used >= len(entries) - 4, rows
    assert errs.max() <= base.TOL, (errs, rows)


def test_vjp_of_a_mixed_engine():
    # the same FP64 adjoint from a mixed-form handle's state, whose dv carries FP32 derivatives
    c = base._state(8)
    out = []
    for form in (abi.FP64, abi.MIXED):
        e = native.Engine(c, precision=form)
        e.initialize(c["pv0"])
        lam = np.random.default_rng(9).normal(size=abi.interior_shape(c["blocks"][0], e.npv))
        out.append(e.residual_vjp([lam])[0][0])
    for v in range(out[0].shape[-1]):
        a, b = out[0][..., v], out[1][..., v]
        assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()

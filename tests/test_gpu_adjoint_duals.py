"""The adjoint's dual-number parts against central differences of the GPU residual (the checks and
the tolerance of test_gpu_adjoint): the fluxes of Roe-M and AUSMPW+ with seven and nine unknowns,
first order and MLP, and the cell sources of the other cavitation models and of a DES length."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, adjoint, native
from tests import test_gpu_adjoint as base

pytestmark = pytest.mark.gpu

# nscheme, nmuscl, nlim, iturb, ncav, ides
VARIANTS = [(2, 2, 8, 0, 1, 0), (3, 2, 8, 0, 1, 0), (2, 2, 8, -2, 1, 0), (3, 2, 8, -2, 1, 0), (2, 0, 0, -2, 1, 0),
            (3, 0, 0, 0, 1, 0), (2, 1, 1, 0, 3, 0), (3, 2, 8, -3, 5, 0), (4, 2, 8, -2, 2, 0), (4, 2, 8, -2, 4, 0),
            (4, 2, 8, 0, 1, 2)]


@pytest.mark.parametrize("variant", VARIANTS, ids=lambda v: "-".join(map(str, v)))
def test_vjp_of_the_dual_parts(variant):
    c = base._state(4)
    for k, v in zip(("nscheme", "nmuscl", "nlim", "iturb", "ncav", "ides"), variant):
        c["cfg"][k] = v
    npv = abi.sizes(c["cfg"])[0]
    c["pv0"] = [np.ascontiguousarray(c["pv0"][0][..., :npv])]
    e = native.Engine(c, precision=abi.FP64)
    e.initialize(c["pv0"])
    s = adjoint.StateSetter(e)
    pv = s.interior(0)
    res = s.residual([pv])[0]
    scale = np.abs(res).reshape(-1, npv).max(axis=0)
    lam = np.random.default_rng(5).normal(size=res.shape) / np.maximum(scale, 1e-300)
    g, _ = e.residual_vjp([lam])
    d = dict(pv=pv, lam=lam, g=g[0])
    entries = base._entries(pv.shape[:-1], npv, 3 * npv, 7)
    used, errs, rows = base._check(lambda p: s.residual([p])[0], d, entries)
    assert used >= len(entries) - 6, rows
    assert errs.max() <= base.TOL, (errs, rows)

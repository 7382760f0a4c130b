"""The FP64 form's face kernels (per-cell planes, reconstruction, three-role flux) against the
CPU oracle's residual: the smallest blocks, extents that leave ragged last CTAs, and every
limiter that bounds its slope by MLP's factor."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native
from tests.helpers import field_err

pytestmark = pytest.mark.gpu

TOL = 1e-9   # the parity tests' residual tolerance


def make(ni, nj, nk, nscheme, nmuscl, nlim, seed=11):
    c = cases.cavitating(scale=8, nscheme=nscheme, fix_cav_clamp=1)
    c["cfg"].update(nmuscl=nmuscl, nlim=nlim)
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0, shear=0.02, seed=seed)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {
        "imin": abi.BC_FARFIELD, "imax": abi.BC_FARFIELD, "jmin": abi.BC_SYMMETRY, "jmax": abi.BC_SYMMETRY,
        "kmin": abi.BC_SYMMETRY, "kmax": abi.BC_SYMMETRY})
    blk = dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])
    rng = np.random.default_rng(seed)
    pv = np.zeros((nk, nj, ni, 7))
    pv[..., 0] = rng.normal(0.0, 2.0e3, (nk, nj, ni))
    pv[..., 1] = c["cfg"]["uref"]
    pv[..., 1:4] += rng.normal(0.0, 0.3, (nk, nj, ni, 3))
    pv[..., 4] = 300.0 + rng.normal(0.0, 0.5, (nk, nj, ni))
    pv[..., 5] = np.where(rng.random((nk, nj, ni)) < 0.4, rng.uniform(0.0, 2e-5, (nk, nj, ni)), 0.0)
    pv[..., 6] = 1e-7
    return dict(c, blocks=[blk], pv0=[pv])


def residuals(c, oracle):
    e, o = native.Engine(c), oracle.Oracle(c)
    e.initialize(c["pv0"])
    o.initialize(c["pv0"])
    return e.residual(0)["res"], o.residual(0)["res"]


@pytest.mark.parametrize("nmuscl,nlim", [(2, 2), (2, 3), (2, 4), (2, 6), (2, 7), (2, 8), (2, 10), (1, 1), (1, 8)])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 7, 5), (65, 3, 4)])
def test_limiters_at_tile_edges(oracle, shape, nmuscl, nlim):
    r, ro = residuals(make(*shape, 4, nmuscl, nlim), oracle)
    assert field_err(r, ro).max() < TOL


@pytest.mark.parametrize("nscheme", [1, 2, 3, 4])
def test_schemes_on_a_ragged_block(oracle, nscheme):
    r, ro = residuals(make(21, 9, 7, nscheme, 2, 8), oracle)
    assert field_err(r, ro).max() < TOL

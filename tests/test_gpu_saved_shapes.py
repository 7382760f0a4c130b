"""Launch shapes saved from an earlier tuning run are taken, whatever fits an SM today: the FP64
form's sweeps from 1 to 8 CTAs per SM, more than are resident included, with the same bits; the
mixed form's to its occupancy limit."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native
from cfd3d_gb300.native import Cfd3dError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.FP64, abi.MIXED])
def test_sweep_ctas_per_sm(precision):
    ni, nj, nk = 131, 67, 71   # more chunks and tiles than any grid below
    c = cases.cavitating(scale=16, fix_cav_clamp=1)
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {f: abi.BC_SYMMETRY for f in ("imin", "imax", "jmin", "jmax", "kmin", "kmax")})
    pv = np.zeros((nk, nj, ni, 7))
    pv[..., 0] = np.random.default_rng(5).normal(0.0, 1.0e3, (nk, nj, ni))
    pv[..., 1] = c["cfg"]["uref"]
    pv[..., 4] = 300.0
    pv[..., 6] = 1e-7
    c = dict(c, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])], pv0=[pv])
    e = native.Engine(c, precision=precision)
    default = e.launch_shapes()
    e.initialize(c["pv0"])
    e.iterate()
    want = e.download(0)["pv"]
    for per in ((1, 3, 5, 8) if precision == abi.FP64 else (1, 2, 3)):
        e.set_launch_shapes((default[0], default[1], per, 1))
        assert e.launch_shapes()[2] == per
        e.initialize(c["pv0"])
        e.iterate()
        assert np.array_equal(e.download(0)["pv"], want), per
    with pytest.raises(Cfd3dError) as ei:
        e.set_launch_shapes((default[0], default[1], 9 if precision == abi.FP64 else 4, 1))
    assert ei.value.code == abi.ERR_ARG
    e.close()

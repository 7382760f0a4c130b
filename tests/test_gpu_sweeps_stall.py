"""A sweep whose waits run out, at shapes with many CTAs waiting at once: the warps leave their
bounded waits as one, the launch ends and is reported, and the handle goes on with the bits of a
fresh one."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native

pytestmark = pytest.mark.gpu


def _case(ni, nj, nk, turb):
    base = cases.adjoint(scale=16) if turb else cases.cavitating(scale=16, fix_cav_clamp=1)
    base["cfg"].update(fix_cav_clamp=1)
    wall = abi.BC_WALL if turb else abi.BC_SYMMETRY
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0, shear=0.02, seed=3)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {
        "imin": abi.BC_FARFIELD, "imax": abi.BC_FARFIELD, "jmin": wall, "jmax": abi.BC_SYMMETRY,
        "kmin": abi.BC_SYMMETRY, "kmax": abi.BC_SYMMETRY})
    npv = abi.sizes(base["cfg"])[0]
    pv = np.zeros((nk, nj, ni, npv))
    pv[..., 0] = np.random.default_rng(5).normal(0.0, 1.0e3, (nk, nj, ni))
    pv[..., 1] = base["cfg"]["uref"]
    pv[..., 4] = 300.0
    pv[..., 6] = 1e-7
    if turb:
        pv[..., 7], pv[..., 8] = base["cfg"]["kinf"], base["cfg"]["oinf"]
    return dict(base, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])], pv0=[pv])


@pytest.mark.parametrize("turb", [False, True])
@pytest.mark.parametrize("shape", [(19, 11, 9), (41, 38, 39)])
@pytest.mark.parametrize("precision", [abi.FP64, abi.MIXED])
def test_waits_that_run_out_end_the_launch(precision, shape, turb):
    c = _case(*shape, turb)
    out = []
    for stall in (False, True):
        e = native.Engine(c, precision=precision)
        e.initialize(c["pv0"])
        if stall:
            for _ in range(3):
                assert e.sweep_stall_test() == abi.ERR_TIMEOUT
            e.initialize(c["pv0"])
        e.iterate()
        out.append(e.download(0)["pv"])
        e.close()
    assert np.array_equal(out[0], out[1])

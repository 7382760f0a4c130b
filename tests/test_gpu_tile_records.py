"""The mixed form's tile records take their face vectors once, at create, through the tile map
that create uploads just before: handle after handle of the same case gives the same bits, for
maps of a few kilobytes and of megabytes, and the first iteration follows the FP64 form's."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 5, 5), (67, 61, 59)])
def test_every_handle_has_the_same_records(shape):
    ni, nj, nk = shape
    base = cases.cavitating(scale=16, fix_cav_clamp=1)
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0, shear=0.02, seed=3)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {
        "imin": abi.BC_FARFIELD, "imax": abi.BC_FARFIELD, "jmin": abi.BC_SYMMETRY, "jmax": abi.BC_SYMMETRY,
        "kmin": abi.BC_SYMMETRY, "kmax": abi.BC_SYMMETRY})
    pv = np.zeros((nk, nj, ni, abi.sizes(base["cfg"])[0]))
    pv[..., 0] = np.random.default_rng(5).normal(0.0, 1.0e3, (nk, nj, ni))
    pv[..., 1] = base["cfg"]["uref"]
    pv[..., 4] = 300.0
    pv[..., 6] = 1e-7
    c = dict(base, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])], pv0=[pv])
    out = []
    for precision in (abi.FP64,) + (abi.MIXED,) * 6:
        e = native.Engine(c, precision=precision)
        e.initialize(c["pv0"])
        before = e.download(0)["pv"]
        e.iterate()
        out.append(e.download(0)["pv"] - before)
        e.close()
    for o in out[2:]:
        assert np.array_equal(o, out[1])
    for v in range(5):   # (a face vector out of its place moves the update by its own size)
        assert np.abs(out[1][..., v] - out[0][..., v]).max() <= 1e-2 * np.abs(out[0][..., v]).max(), v

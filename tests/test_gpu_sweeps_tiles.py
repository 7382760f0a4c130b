"""The mixed form's tile sweeps at the shapes where a tile's entries can go to the wrong cell
or step: blocks smaller than a tile, whole tiles, ragged ends in each direction, seven and
nine variables.  Reference: the FP64 form's sweeps, which share no code with them."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native

pytestmark = pytest.mark.gpu

# The update of one iteration is linear in the FP32 roundings of the residual, the diagonal
# block and the products: 6e-8 each, some hundred of them per cell, over up to 60 cells of a
# chain whose terms cancel to about a tenth: 4e-3 of the largest change.  An entry that goes
# astray is of the order of the change itself.
TOL = 1e-2


@pytest.mark.parametrize("turb", [False, True])
@pytest.mark.parametrize("shape", [(3, 3, 3), (8, 8, 4), (16, 8, 9), (9, 17, 5), (35, 7, 13)])
def test_tile_sweeps_follow_the_fp64_form(shape, turb):
    ni, nj, nk = shape
    base = cases.adjoint(scale=16) if turb else cases.cavitating(scale=16, fix_cav_clamp=1)
    base["cfg"].update(fix_cav_clamp=1)
    wall = abi.BC_WALL if turb else abi.BC_SYMMETRY
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0, shear=0.02, seed=3)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {
        "imin": abi.BC_FARFIELD, "imax": abi.BC_FARFIELD, "jmin": wall, "jmax": abi.BC_SYMMETRY,
        "kmin": abi.BC_SYMMETRY, "kmax": abi.BC_SYMMETRY})
    npv = abi.sizes(base["cfg"])[0]
    rng = np.random.default_rng(5)
    pv = np.zeros((nk, nj, ni, npv))
    pv[..., 0] = rng.normal(0.0, 1.0e3, (nk, nj, ni))
    pv[..., 1] = base["cfg"]["uref"]
    pv[..., 1:4] += rng.normal(0.0, 0.2, (nk, nj, ni, 3))
    pv[..., 4] = 300.0
    pv[..., 6] = 1e-7
    if turb:
        pv[..., 7], pv[..., 8] = base["cfg"]["kinf"], base["cfg"]["oinf"]
    c = dict(base, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])], pv0=[pv])
    out = []
    for precision in (abi.FP64, abi.MIXED, abi.MIXED):
        e = native.Engine(c, precision=precision)
        e.initialize(c["pv0"])
        before = e.download(0)["pv"]
        e.iterate()
        out.append(e.download(0)["pv"] - before)
        e.close()
    assert np.array_equal(out[1], out[2])   # whichever CTA took which tile
    for v in [0, 1, 2, 3, 4] + ([7, 8] if turb else []):
        scale = np.abs(out[0][..., v]).max()
        assert np.abs(out[1][..., v] - out[0][..., v]).max() <= TOL * scale, v

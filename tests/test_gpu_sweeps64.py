"""The FP64 form's dataflow sweeps at the shapes where a chunk of a hyperplane, or a warp's
share of it, can go wrong: planes smaller than a chunk, planes of many chunks with ragged
ends, seven and nine variables.  Reference: one launch per hyperplane, the same arithmetic
per cell."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turb", [False, True])
@pytest.mark.parametrize("shape", [(3, 3, 3), (3, 40, 3), (35, 5, 4), (41, 38, 39)])
def test_dataflow_equals_hyperplanes(monkeypatch, shape, turb):
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
    for mode in ("planes", "dataflow"):
        monkeypatch.setenv("CFD3D_SWEEP", mode)
        e = native.Engine(c)
        e.initialize(c["pv0"])
        e.iterate()
        out.append(e.download(0)["pv"])
        e.close()
    scale = np.abs(out[0]).reshape(-1, npv).max(axis=0)
    assert (np.abs(out[0] - out[1]).reshape(-1, npv).max(axis=0) <= 1e-12 * scale).all()

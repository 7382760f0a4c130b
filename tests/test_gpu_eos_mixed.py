"""The mixed form's cell EOS in passes (liquid, listed vapour, mixture), as the update runs it,
against the same EOS in one piece, as an upload runs it: liquid cells, cells with metastable
and with stable vapour and all three mixed, stiffened water, ragged counts."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fluid", [1, 2])
@pytest.mark.parametrize("kind", ["liquid", "metastable", "stable", "all"])
@pytest.mark.parametrize("shape", [(3, 3, 3), (37, 7, 5)])
def test_passes_equal_the_whole(shape, kind, fluid):
    ni, nj, nk = shape
    base = cases.cavitating(scale=16, fix_cav_clamp=1)
    # a step too short to move the state: the update's EOS sees the states made here
    base["cfg"].update(cfl=1e-7, fluid=fluid, ncav=0)
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0, shear=0.02, seed=3)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {f: abi.BC_SYMMETRY for f in ("imin", "imax", "jmin", "jmax", "kmin", "kmax")})
    npv = abi.sizes(base["cfg"])[0]
    rng = np.random.default_rng(7)
    pv = np.zeros((nk, nj, ni, npv))
    pick = {"liquid": 0, "metastable": 1, "stable": 2}.get(kind)
    which = rng.integers(0, 3, (nk, nj, ni)) if pick is None else np.full((nk, nj, ni), pick)
    p = np.where(which == 2, 2.0e3, 6.0e4) + rng.normal(0.0, 1.0e2, (nk, nj, ni))   # saturation at 3.5e3 Pa
    pv[..., 0] = p - base["cfg"]["pref"]
    pv[..., 1] = base["cfg"]["uref"]
    pv[..., 4] = 300.0 + rng.normal(0.0, 1.0, (nk, nj, ni))
    pv[..., 5] = np.where(which == 0, 0.0, rng.uniform(0.01, 0.3, (nk, nj, ni)))
    pv[..., 6] = 1e-7
    c = dict(base, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])], pv0=[pv])
    e = native.Engine(c, precision=abi.MIXED)
    e.initialize(c["pv0"])
    e.iterate()
    a = e.download(0)
    e.close()
    other = pv.copy()
    other[..., 4] += 1.0
    e = native.Engine(c, precision=abi.MIXED)
    e.initialize([other])
    e.upload_primitives(0, pv=a["pv"])
    b = e.download(0)
    e.close()
    inner = (slice(3, 3 + nk), slice(3, 3 + nj), slice(3, 3 + ni))
    assert np.array_equal(a["pv"][inner], b["pv"][inner])
    for v in range(18):
        x, y = a["dv"][inner][..., v], b["dv"][inner][..., v]
        # rho and h to FP64 sums of a few terms; the rest is FP32, some thirty roundings
        tol = 1e-14 * np.abs(y) if v < 2 else 2e-6 * np.abs(y).max()
        assert (np.abs(x - y) <= tol).all(), v
    for v in range(2):
        x, y = a["tv"][inner][..., v], b["tv"][inner][..., v]
        assert (np.abs(x - y) <= 2e-6 * np.abs(y).max()).all(), v

"""The sweeps where vapour and gas vary from cell to cell: the mass fractions' columns of D^-1 and
of the neighbours' products, which a vapour-free or uniform state multiplies by nothing.  The FP64
form's first iteration against the CPU oracle's, which shares no code with it, and the mixed form's
against the FP64 form's, every variable, ragged blocks, seven and nine unknowns."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native
from tests.helpers import field_err, interior

pytestmark = pytest.mark.gpu

# The change of one iteration is linear in the residual, which the two agree on to 1e-9 of each
# variable's largest (the parity tests' tolerance); D^-1 takes differences of terms up to a thousand
# times its result (1 / c^2 against the preconditioned 1 / V^2).  An error in a coefficient is of
# the order of the change.
TOL64 = 1e-6
# as for the tile sweeps: FP32 roundings, some hundred a cell, over a chain of cells
TOL_MIXED = 1e-2
SHAPES = [(3, 3, 3), (9, 17, 5), (35, 5, 4), (16, 8, 9)]


def make(ni, nj, nk, turb):
    base = cases.adjoint(scale=16) if turb else cases.cavitating(scale=16, fix_cav_clamp=1)
    base["cfg"].update(fix_cav_clamp=1)
    wall = abi.BC_WALL if turb else abi.BC_SYMMETRY
    xyz = cases.box_nodes(ni, nj, nk, 2.0, 1.0, 1.0, shear=0.02, seed=3)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {
        "imin": abi.BC_FARFIELD, "imax": abi.BC_FARFIELD, "jmin": wall, "jmax": abi.BC_SYMMETRY,
        "kmin": abi.BC_SYMMETRY, "kmax": abi.BC_SYMMETRY})
    npv = abi.sizes(base["cfg"])[0]
    rng = np.random.default_rng(5)
    size = (nk, nj, ni)
    pv = np.zeros(size + (npv,))
    pv[..., 0] = rng.normal(0.0, 1.0e3, size)
    pv[..., 1] = base["cfg"]["uref"]
    pv[..., 1:4] += rng.normal(0.0, 0.2, size + (3,))
    pv[..., 4] = 300.0 + rng.normal(0.0, 0.5, size)
    pv[..., 5] = np.where(rng.random(size) < 0.3, 0.0, 10.0 ** rng.uniform(-5, -2, size))
    pv[..., 6] = 10.0 ** rng.uniform(-6, -3, size)
    if turb:
        pv[..., 7] = base["cfg"]["kinf"] * rng.uniform(0.5, 2.0, size)
        pv[..., 8] = base["cfg"]["oinf"] * rng.uniform(0.5, 2.0, size)
    return dict(base, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])], pv0=[pv])


def change(e, c):
    e.initialize(c["pv0"])
    e.iterate()
    return interior(e.download(0)["pv"]) - c["pv0"][0]


@pytest.mark.parametrize("mode", ["dataflow", "planes"])
@pytest.mark.parametrize("turb", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_against_the_oracle(oracle, monkeypatch, shape, turb, mode):
    c = make(*shape, turb)
    monkeypatch.setenv("CFD3D_SWEEP", mode)
    e = native.Engine(c)
    got = change(e, c)
    e.close()
    o = oracle.Oracle(c)
    o.initialize(c["pv0"])
    o.iterate()
    want = interior(o.get_state(0)["pv"]) - c["pv0"][0]
    assert np.abs(want[..., 5]).max() > 1e-6 and np.abs(want[..., 6]).max() > 1e-9
    assert (field_err(got, want) < TOL64).all(), field_err(got, want)


@pytest.mark.parametrize("turb", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_mixed_against_fp64(shape, turb):
    c = make(*shape, turb)
    out = []
    for precision in (abi.FP64, abi.MIXED, abi.MIXED):
        e = native.Engine(c, precision=precision)
        out.append(change(e, c))
        e.close()
    assert np.array_equal(out[1], out[2])   # whichever CTA took which tile
    assert (field_err(out[1], out[0]) < TOL_MIXED).all(), field_err(out[1], out[0])

"""Where the FP64 form keeps the scratch planes of its face reconstruction: an allocation for
three directions (small cases), the sweep records' memory (larger ones), an allocation for one
direction (many cells in blocks that are mostly padding).  Each gives the oracle's residual, before
and after sweeps have used the records, and a large case holds no more memory than its state,
face and sweep arrays."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native
from tests import test_gpu_adjoint as base
from tests.helpers import field_err
from tests.test_gpu_faces64 import TOL, make

pytestmark = pytest.mark.gpu


# padded cells over 1.28e8 / (3 x 5 x 7 x 8) = 152380 take one direction at a time
@pytest.mark.parametrize("shape", [(21, 9, 7), (61, 47, 43), (3, 3, 1900)])
def test_residual_wherever_the_planes_lie(oracle, shape):
    c = make(*shape, 4, 2, 8)
    e, o = native.Engine(c), oracle.Oracle(c)
    e.initialize(c["pv0"])
    o.initialize(c["pv0"])
    ro = o.residual(0)["res"]
    assert field_err(e.residual(0)["res"], ro).max() < TOL
    e.iterate()
    e.initialize(c["pv0"])
    assert field_err(e.residual(0)["res"], ro).max() < TOL
    e.close()


def test_memory_of_a_large_case():
    torch = pytest.importorskip("torch")
    warm = native.Engine(cases.make("plain_small", scale=8))   # the context and its modules
    warm.initialize(None)
    warm.iterate()
    ni, nj, nk = 131, 97, 101
    c = base._state(4)
    c["cfg"].update(nsteady=2, dt_phy=1e-3)
    xyz = cases.box_nodes(ni, nj, nk, 1.0, 1.0, 1.0)
    bc = cases.face_patches(ni + 1, nj + 1, nk + 1, {
        "imin": abi.BC_FARFIELD, "imax": abi.BC_FARFIELD, "jmin": abi.BC_SYMMETRY, "jmax": abi.BC_SYMMETRY,
        "kmin": abi.BC_SYMMETRY, "kmax": abi.BC_SYMMETRY})
    c = dict(c, blocks=[dict(imax=ni + 1, jmax=nj + 1, kmax=nk + 1, xyz=xyz, bc=bc, con=[])])
    free = torch.cuda.mem_get_info()[0]
    e = native.Engine(c, precision=abi.FP64)
    held = free - torch.cuda.mem_get_info()[0]
    e.close()
    warm.close()
    padded, cells = (ni + 6) * (nj + 6) * (nk + 6), ni * nj * nk
    # planes of the padded cells: pv 9, dv 18, tv 3, metrics 14, residual 9, icav 4, itt 4, omega
    # bound 1, dt 1, rcav 2, history 18, dq and the sweeps' right-hand side 9 each, fluxes 27 + 27;
    # the cells' positions; per cell seven indices and the 61-value records.  Forty allocations
    # round up to 2 MB each, and the face scratch would add 360 B per padded cell (522 MB)
    want = padded * (8 * 155 + 4) + cells * (28 + 8 * 61)
    assert held <= want + 40 * (2 << 20), (held, want)

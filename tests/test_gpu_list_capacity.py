"""The mixed form's state lists hold 32-bit entries, two per face of a direction: a grid with more
is refused by name before any allocation, and the largest extents below it get past that check."""
import ctypes as C

import numpy as np
import pytest

from cfd3d_gb300 import abi, cases, native

pytestmark = pytest.mark.gpu


def _create(imax, jmax, kmax):
    # (the nodes are not read: such a grid is refused for its size or for memory)
    cfg = abi.config_from_dict(dict(cases.cavitating(scale=16)["cfg"], precision=abi.MIXED))
    nodes = np.zeros(3)
    blk = (abi.BlockDesc * 1)()
    blk[0].imax, blk[0].jmax, blk[0].kmax = imax, jmax, kmax
    blk[0].xyz = nodes.ctypes.data_as(C.POINTER(C.c_double))
    h = C.c_void_p()
    rc = native.lib().cfd3d_create(C.byref(cfg), 1, blk, C.byref(h))
    msg = native.lib().cfd3d_last_error(h).decode()
    native.lib().cfd3d_destroy(h)
    return rc, msg


@pytest.mark.parametrize("shape", [(1025, 1025, 1025), (65, 4097, 4097), (4097, 4097, 65)])
def test_more_states_than_entries(shape):
    # imax (jmax - 1)(kmax - 1) faces and more of one direction: over 2^30
    rc, msg = _create(*shape)
    assert rc == abi.ERR_ARG and "lists" in msg


def test_the_largest_below_is_a_matter_of_memory():
    # 1.08e9 padded cells: pv, dv, tv and the metrics alone take 346 GB
    rc, msg = _create(1021, 1021, 1021)
    assert rc == abi.ERR_NOMEM

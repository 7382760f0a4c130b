"""Device memory: calls that find none left report it and leave the handle usable."""
import numpy as np
import pytest

from cfd3d_gb300 import abi, native
from cfd3d_gb300.native import Cfd3dError
from tests import test_gpu_adjoint as base

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _fill(leave):
    """all of the device's free memory but about `leave` bytes"""
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty((free - leave) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda")


# 64^3 cells in 70^3: 25 MB for each of the cotangent and the gradient, 27 MB for dv and tv; a
# mixed-form handle then needs the face states and 123 MB of reconstruction planes
@pytest.mark.parametrize("precision,leave", [(abi.FP64, 40 * MB), (abi.MIXED, 40 * MB), (abi.MIXED, 190 * MB)])
def test_adjoint_after_out_of_memory(precision, leave):
    import torch
    c = base._state(1)
    lam = np.random.default_rng(9).normal(size=abi.interior_shape(c["blocks"][0], 9))
    e = native.Engine(c, precision=precision)
    e.initialize(c["pv0"])
    hold = _fill(leave)
    for _ in range(2):
        with pytest.raises(Cfd3dError) as ei:
            e.residual_vjp([lam])
        assert ei.value.code == abi.ERR_NOMEM
    del hold
    torch.cuda.empty_cache()
    g = e.residual_vjp([lam])[0][0]
    e.close()
    f = native.Engine(c, precision=precision)
    f.initialize(c["pv0"])
    want = f.residual_vjp([lam])[0][0]
    f.close()
    for v in range(9):   # (sums by atomics, in any order)
        assert np.abs(g[..., v] - want[..., v]).max() <= 1e-10 * np.abs(want[..., v]).max()


def test_a_failed_create_leaves_the_other_calls_alone():
    import torch
    c = base._state(1)
    rng = np.random.default_rng(3)
    p, t = rng.uniform(2e3, 3e5, 5000), rng.uniform(280.0, 320.0, 5000)
    y1, y2 = rng.uniform(0.0, 0.5, 5000), np.full(5000, 1e-7)
    want = native.eos_eval(p, t, y1, y2, prop=True)
    for points in (5, 5000):   # through the static buffer, through an allocation
        hold = _fill(40 * MB)
        with pytest.raises(Cfd3dError) as ei:
            native.Engine(c, precision=abi.FP64)
        assert ei.value.code == abi.ERR_NOMEM
        del hold
        torch.cuda.empty_cache()
        got = native.eos_eval(p[:points], t[:points], y1[:points], y2[:points], prop=True)
        assert np.array_equal(got[0], want[0][:points]) and np.array_equal(got[1], want[1][:points])
    hold = _fill(40 * MB)
    with pytest.raises(Cfd3dError):
        native.Engine(c, precision=abi.MIXED)
    del hold
    torch.cuda.empty_cache()
    e = native.Engine(c, precision=abi.MIXED)
    e.initialize(c["pv0"])
    assert np.all(np.isfinite(e.iterate()[1]))
    e.close()


def test_memory_of_the_mixed_adjoint():
    import torch
    c = base._state(1)
    lam = np.random.default_rng(9).normal(size=abi.interior_shape(c["blocks"][0], 9))
    e = native.Engine(c, precision=abi.MIXED)
    e.initialize(c["pv0"])
    e.iterate()
    small = native.Engine(base._state(4), precision=abi.MIXED)   # the kernels' modules and stacks
    small.initialize(None)
    small.residual_vjp([np.ones((16, 16, 16, 9))])
    free = torch.cuda.mem_get_info()[0]
    e.residual_vjp([lam])
    held = free - torch.cuda.mem_get_info()[0]
    e.close()
    small.close()
    # planes of 70^3 cells: cotangent and gradient 9 each, dv and tv 10, one direction's face states
    # 9, five reconstruction planes a variable; seven allocations round up to 2 MB each
    assert held <= 8 * 70 ** 3 * (9 + 9 + 10 + 9 + 45) + 7 * 2 * MB, held / MB


@pytest.mark.parametrize("precision,scale", [(abi.MIXED, 1), (abi.FP64, 2)])
def test_create_with_little_memory_takes_the_directions_in_turn(precision, scale):
    import torch
    c = base._state(scale)

    def run():
        e = native.Engine(c, precision=precision)
        e.initialize(c["pv0"])
        for it in range(2):
            e.iterate(1, it + 1, 0.0)
        pv = e.download(0)["pv"]
        e.close()
        return pv

    want = run()
    free = torch.cuda.mem_get_info()[0]
    e = native.Engine(c, precision=precision)
    full = free - torch.cuda.mem_get_info()[0]
    e.close()
    # the other directions' scratch is 78 MB (64^3 cells, mixed) and 39 MB (32^3, FP64)
    hold = _fill(full - 12 * MB)
    e = native.Engine(c, precision=precision)
    del hold
    torch.cuda.empty_cache()
    e.initialize(c["pv0"])
    for it in range(2):
        e.iterate(1, it + 1, 0.0)
    assert np.array_equal(e.download(0)["pv"], want)
    e.close()

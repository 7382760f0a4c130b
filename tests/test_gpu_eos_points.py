"""Pointwise EOS at the counts where its route changes: packed copies, the static buffer's
last point, an allocation.  A point's values do not depend on the route."""
import numpy as np
import pytest

from cfd3d_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fluid,prop", [(2, True), (2, False), (1, True)])
def test_points_do_not_depend_on_the_route(fluid, prop):
    n = native.EOS_NOALLOC_MAX + 1
    rng = np.random.default_rng(3)
    p, t = rng.uniform(2e3, 3e5, n), rng.uniform(280.0, 320.0, n)
    y1 = rng.uniform(0.0, 0.5, n) * (rng.uniform(size=n) < 0.5)
    y2 = 10.0 ** rng.uniform(-7, -3, n)
    dv, tv = native.eos_eval(p, t, y1, y2, fluid=fluid, prop=prop)
    per_point = 20 if prop else 18   # results of a point; 8192 of them are packed at most
    for m in (1, 31, 33, 8192 // per_point, 8192 // per_point + 1, n - 1):
        a, b = native.eos_eval(p[:m], t[:m], y1[:m], y2[:m], fluid=fluid, prop=prop)
        assert np.array_equal(a, dv[:m]), m
        assert np.array_equal(b, tv[:m]), m

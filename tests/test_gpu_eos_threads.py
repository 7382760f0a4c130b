"""Pointwise EOS from several host threads at once: calls of one context share the static buffer
and take turns, larger ones have their own memory; every call has its own points' values."""
import threading

import numpy as np
import pytest

from cfd3d_gb300 import native

pytestmark = pytest.mark.gpu


def test_threads_have_their_own_values():
    sizes = (3, 200, 777, native.EOS_NOALLOC_MAX, native.EOS_NOALLOC_MAX + 1)
    pts = []
    for q, n in enumerate(sizes):
        rng = np.random.default_rng(q)
        pts.append((rng.uniform(2e3, 3e5, n), rng.uniform(280.0, 320.0, n),
                    rng.uniform(0.0, 0.5, n) * (rng.uniform(size=n) < 0.5), 10.0 ** rng.uniform(-7, -3, n)))
    want = [native.eos_eval(*p, prop=True) for p in pts]
    bad = []

    def work(q):
        for _ in range(30):
            for f in (native.eos_eval, native.eos_eval_noalloc):
                if f is native.eos_eval_noalloc and sizes[q] > native.EOS_NOALLOC_MAX:
                    continue
                dv, tv = f(*pts[q], prop=True)
                if not (np.array_equal(dv, want[q][0]) and np.array_equal(tv, want[q][1])):
                    bad.append(q)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad

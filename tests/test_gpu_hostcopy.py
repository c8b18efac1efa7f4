"""Field copies large enough for the pinned ring of hostcopy.cu (above 32 MB, not
a multiple of its 512 KB slots) come back bit for bit, from one thread and from
two contexts in two threads at once, and again after the last context has given
the ring back; and contexts of several threads, created at once."""
import threading

import numpy as np
import pytest

from fopis_b200 import RootGrid, _abi, config
from fopis_b200.config import SpeciesInfo, make_params, plasma_units

pytestmark = pytest.mark.gpu


def grid(n):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, 1)]
    p, norm = make_params((n, n + 1, n - 2), "DDDDDD", dx, dt, sp)
    return RootGrid(config.SimConfig(params=p, norm=norm, species=sp))


def round_trips(n, seed, failed):
    g = grid(n)
    for k in range(3):
        a = np.random.default_rng(seed + k).standard_normal(g.shape)
        g.set_field(_abi.FIELD_RHO0, a)
        if not np.array_equal(g.getRho(), a):
            failed.append((n, k))
    g.close()


@pytest.mark.parametrize("sizes", [(161,), (161, 170)])
def test_large_fields_round_trip(gpu_available, sizes):
    failed = []
    in_threads([lambda i=i, n=n: round_trips(n, 10 * i, failed) for i, n in enumerate(sizes)])
    assert not failed


def in_threads(calls):
    """Runs the calls at once; an exception in one of them fails the test."""
    raised = []

    def guarded(call):
        try:
            call()
        except Exception as e:
            raised.append(e)

    threads = [threading.Thread(target=guarded, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not raised, raised


def test_contexts_of_several_threads(gpu_available):
    """Threads that create, use and close contexts of their own while others record their solve graphs."""
    def work(n):
        for k in range(6):
            g = grid(n)
            a = np.random.default_rng(k).standard_normal(g.shape)
            g.set_field(_abi.FIELD_RHO0, a)
            assert g.solvePoisson() == 0 and np.array_equal(g.getRho(), a)
            g.close()

    in_threads([lambda n=n: work(n) for n in (9, 12, 17, 20, 33, 34)])

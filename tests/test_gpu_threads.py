"""Contexts of different sizes in several host threads: a kernel's dynamic shared memory differs between them, and what
one call sets for its launch must not reach another's."""
import threading

import numpy as np
import pytest

from spring_b200 import synthetic as S
from spring_b200.api import from_crystal

pytestmark = pytest.mark.gpu


def _cell(nb):
    b = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0], [.5, .5, .5]], float)[:nb]
    cr = S.Crystal("cell", 4.0 * np.eye(3), b, np.ones(nb, np.int32), np.linspace(20.0, 60.0, nb))
    S.make_fc2(cr)
    S.make_fc3(cr)
    return cr


def _together(calls, repeat):
    """Every call `repeat` times, each in its own thread; results equal to those of the call alone."""
    alone = [np.array(f()) for f in calls]
    errors, start = [], threading.Barrier(len(calls))

    def work(f, ref):
        try:
            start.wait()
            for _ in range(repeat):
                np.testing.assert_allclose(np.array(f()), ref, rtol=1e-9, atol=1e-12 * np.abs(ref).max())
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_iterative_kappa_in_threads():
    ctxs = [from_crystal(S.build("rocksalt2"), (n, n, n), [300.0])[0] for n in (5, 10)]
    _together([lambda c=c: c.kappa_iter(eps_k=1e-9, max_iter=25)["kappa"] for c in ctxs], 60)
    for c in ctxs:
        c.close()


def test_linewidths_of_different_cells_in_threads():
    ctxs = [from_crystal(_cell(nb), (3, 2, 2), [300.0])[0] for nb in (3, 4, 5)]
    ctxs.append(from_crystal(S.build("rocksalt8"), (2, 2, 2), [300.0])[0])
    _together([lambda c=c: c.linewidth3(1, c.nq0, "gauss", 1.5)[0] for c in ctxs], 200)
    for c in ctxs:
        c.use_generic_v3(True)
    _together([lambda c=c: c.linewidth3(1, c.nq0, "gauss", 1.5)[0] for c in ctxs], 200)
    for c in ctxs:
        c.close()

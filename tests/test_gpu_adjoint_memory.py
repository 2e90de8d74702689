"""The adjoint's device memory, which the handle keeps between runs: runs of
other lengths and checkpoint counts in between, and other handles' runs at the
same time, change nothing to the last bit."""
import threading

import numpy as np
import pytest

import adjoint_cases as ac
from dugks_b200 import lib as dl

pytestmark = pytest.mark.gpu


def _run(s, c, steps, snapshots):
    hw, fw, _ = ac.objective_weights(c)
    r = s.adjoint(steps, c.dt, hw, fw, max_snapshots=snapshots)
    return np.concatenate([[r["J"], r["dmu"]], np.ravel(r["dT_b"]), np.ravel(r["dU_b"])])


@pytest.mark.parametrize("which", ["cavity", "farfield"])
def test_runs_in_any_order_agree(which):
    c = ac.cases()[which]
    fresh = [_run(dl.Solver(c), c, n, k) for n, k in ((5, 2), (3, 3))]
    s = dl.Solver(c)
    for n, k, want in ((5, 2, fresh[0]), (3, 3, fresh[1]), (5, 2, fresh[0]), (5, 2, fresh[0])):
        assert np.array_equal(_run(s, c, n, k), want)
        s.boundary_fluxes(c.dt)


def test_two_handles_on_two_threads():
    c = ac.cases()["cavity"]
    want = _run(dl.Solver(c), c, 5, 2)
    got = [None, None]

    def work(i):
        s = dl.Solver(c)
        got[i] = [_run(s, c, 5, 2) for _ in range(4)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for rs in got:
        assert all(np.array_equal(r, want) for r in rs)

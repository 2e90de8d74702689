"""A 3-D handle with KInner 0 that carried h for a while (a nonzero h~ was
loaded) and starts again from macros: h is identically zero once more, and
the adjoint, the objective and the boundary fluxes see none of the old run's
h, to the last bit."""
import numpy as np
import pytest

import adjoint_cases as ac
from dugks_b200 import case as cs
from dugks_b200 import lib as dl

pytestmark = pytest.mark.gpu


def _answers(s, c):
    hw, fw, _ = ac.objective_weights(c)
    r = s.adjoint(3, c.dt, hw, fw, max_snapshots=2)
    flux = s.boundary_fluxes(c.dt)
    J = s.objective(2, c.dt, hw, fw)[0]
    return np.concatenate([[r["J"], r["dmu"], J], np.ravel(r["dT_b"]), np.ravel(r["dU_b"]), np.ravel(flux)])


@pytest.mark.parametrize("which", ["cube", "ball"])
def test_h_of_an_earlier_run_leaves_no_trace(which):
    c = cs.cube_case(4, 6) if which == "cube" else cs.ball_case(2, 3, 1.12, 6, kn=0.1, mach=0.5)
    want = _answers(dl.Solver(c), c)
    s = dl.Solver(c)
    s.step(1, c.dt)
    g, _ = s.state()
    s.set_state(g, 0.01 * c.gas["R"] * 273.0 * g, c.dt)
    s.step(2, c.dt)
    s.set_macros(c.rho0, c.U0, c.T0)
    assert np.array_equal(_answers(s, c), want)

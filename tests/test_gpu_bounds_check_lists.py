"""The bounds-checked build on the tables of the streaming kernels: the cell
order of a state that is set and read, the caller's face order, the rows of
the DV set and the list of tangential pairs with its places (FP32).  No check
fires, and the checked build gives what the normal build gives, to an ulp."""
import numpy as np
import pytest

from dugks_b200 import case as cs
from dugks_b200 import lib as dl
from dugks_b200 import quadrature

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [dl.FP64, dl.FP32C])
@pytest.mark.parametrize("n_dv", [9, 33])
def test_checked_state_order_and_tangential_pairs(n_dv, precision):
    c = cs.cavity_case(9, 8, flatten=False)
    c.xis, c.weights = quadrature.newton_cotes(1600.0, n_dv)
    c.xi_max = 1600.0
    c.flatten()
    # what an ulp of the storage type is of each quantity's natural scale
    C = np.sqrt(2.0 * c.gas["R"] * 273.0)
    scale = {"rho": c.rho0.max(), "U": C, "T": 273.0, "q": c.rho0.max() * C**3}
    tol = 1e-13 if precision == dl.FP64 else 1e-6
    out = []
    for path in (None, dl.CHECK_LIB_PATH):
        s = dl.Solver(c, precision=precision, lib_path=path)
        s.step(2, c.dt)                        # raises DugksError if a check fired
        s.set_state(*s.state(), c.dt, s.step_record())
        s.step(2, c.dt)
        out.append((s.macros(), s.face_macros(), *s.state()))
    (ma, fa, ga, ha), (mb, fb, gb, hb) = out
    for a, b in ((ma, mb), (fa, fb)):
        for k in a:
            assert np.abs(a[k] - b[k]).max() <= tol * scale[k], k
    for a, b in ((ga, gb), (ha, hb)):
        assert np.abs(a - b).max() <= tol * np.abs(a).max()

"""(entity, DV) arrays of 2^32 elements and more, where the step's kernels
take 64-bit offsets: one handle against the two halves of its DV set, whose
arrays stay below that size and take 32-bit offsets.  Start fields vary from
cell to cell, so that an element of another cell or DV shows."""
import numpy as np
import pytest

import oracle_bind as ob
from dugks_b200 import case as cs
from dugks_b200 import lib as dl
from dugks_b200 import shard as sh

pytestmark = pytest.mark.gpu

# the sums over the DVs in another order: FP64 rounding, and FP32 storage of
# the state after it (the mixed-precision path's bound against the oracle)
TOL = {dl.FP64: 1e-12, dl.FP32C: 5e-6}


def _case(D, listed):
    c = cs.cube_case(18, 6, kn=0.1, flatten=False) if D == 3 else cs.cavity_case(730, 6, flatten=False)
    x = np.linspace(-1600.0, 1600.0, 64)
    w = np.full(64, x[1] - x[0])
    w[0] = w[-1] = 0.5 * w[0]
    c.xis, c.weights, c.xi_max = x, w, 1600.0
    if listed:
        c.dv_xi, c.dv_w = c.dv_set()
    r = np.random.default_rng(D)
    n = c.n_cells
    c.rho0 = c.rho0 * r.uniform(0.9, 1.1, n)
    c.T0 = c.T0 * r.uniform(0.9, 1.1, n)
    c.U0 = r.uniform(-40.0, 40.0, (n, 3)) * ([1, 1, 1] if D == 3 else [1, 1, 0])
    return c.flatten()


@pytest.mark.parametrize("D,listed,precision", [(3, False, dl.FP64), (3, False, dl.FP32C), (3, True, dl.FP32C),
                                                (2, False, dl.FP32C)])
def test_whole_set_and_its_halves_agree(D, listed, precision):
    c = _case(D, listed)
    faces = (c.flat["n_internal"] + c.flat["n_boundary"] + 31) // 32 * 32
    assert faces * c.n_dv >= 1 << 32 > faces * c.n_dv // 2 + 1024
    s = dl.Solver(c, precision=precision)
    s.step(2, c.dt)
    got = s.macros()
    s.close()
    halves = [dl.Solver(c, precision=precision, shard=dl.shard(r, 2)) for r in range(2)]
    sh.step_local(halves, 2, c.dt)
    want = halves[0].macros()
    for h in halves:
        h.close()
    errs = ob.macro_errors(got, want, c.gas["R"])
    assert max(errs.values()) <= TOL[precision], errs

"""Edges of the streaming kernels' blocks against the CPU oracle: rows of DVs
that are no multiple of the groups of four and the blocks of eight, rows of
more than 32 DVs (two segments), cell and face counts around the blocks of 32
entities, exactly tangential pairs in every remainder; and the state's copies
between the caller's order and the device's.

Tolerances: FP64 as in the parity tests, 1e-10 relative L2 (sums of another
order); FP32 storage 5e-6 as there.  A state read back is the one loaded,
FP32 storage to one rounding of the deviation: 2^-24 (|g| + |ref|) and the
FP64 sum's own 2^-53, both under 2^-22 of the largest value."""
import numpy as np
import pytest

import oracle_bind as ob
from dugks_b200 import case as cs
from dugks_b200 import lib as dl
from dugks_b200 import quadrature

pytestmark = pytest.mark.gpu

TOL = {dl.FP64: 1e-10, dl.FP32C: 5e-6}


def _newton_cotes(n, n_dv):
    c = cs.cavity_case(n, 8, flatten=False)
    c.xis, c.weights = quadrature.newton_cotes(1600.0, n_dv)
    c.xi_max = 1600.0
    c.flatten()
    return c


@pytest.mark.parametrize("precision", [dl.FP64, dl.FP32C])
@pytest.mark.parametrize("n,n_dv", [(3, 5), (6, 9), (9, 13), (9, 33), (11, 37), (33, 17)])
def test_row_remainders_and_tangential_pairs(n, n_dv, precision):
    c = _newton_cotes(n, n_dv)
    gpu, orc = dl.Solver(c, precision=precision), ob.Oracle(c)
    for _ in range(2):
        gpu.evolution(c.dt)
        orc.evolution(c.dt)
    tol = TOL[precision]
    assert max(ob.macro_errors(gpu.macros(), orc.macros(), c.gas["R"]).values()) <= tol
    if precision == dl.FP64:
        assert max(ob.macro_errors(gpu.face_macros(), orc.face_macros(), c.gas["R"]).values()) <= tol
    for a, b in zip(gpu.state(), orc.state()):
        assert ob.rel_l2(a, b) <= tol


@pytest.mark.parametrize("precision", [dl.FP64, dl.FP32C])
@pytest.mark.parametrize("n,n_dv", [(3, 6), (8, 8), (13, 10), (33, 6)])
def test_state_round_trip(n, n_dv, precision):
    c = cs.cavity_case(n, n_dv)
    s = dl.Solver(c, precision=precision)
    g0, h0 = s.state()
    rng = np.random.default_rng(n)
    g, h = g0 * rng.uniform(0.9, 1.1, g0.shape), h0 * rng.uniform(0.9, 1.1, h0.shape)
    s.set_state(g, h, c.dt)
    cells = np.array([0, c.n_cells // 2, c.n_cells - 1], dtype=np.int32)
    for a, b, df in zip(s.state(), (g, h), s.df(cells)):
        if precision == dl.FP64:
            assert np.array_equal(a, b)
        else:
            assert np.abs(a - b).max() <= 2.0**-22 * np.abs(b).max()
        assert np.array_equal(np.asarray(df).reshape(len(cells), -1), a[:, cells].T)

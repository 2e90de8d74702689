"""Symmetry patches whose faces are not all parallel to the first one.

The DVs a face takes from the mirror side are chosen by the patch's first
face, the ones it reconstructs by its own area vector, so on a tilted face
some DVs are neither: they carry no distribution function from step to step.
A run that is saved and continued on a fresh handle is then, bit for bit, the
run that went on."""
import numpy as np
import pytest

from dugks_b200 import case as cs
from dugks_b200 import lib as dl

pytestmark = pytest.mark.gpu


def _tilted(kind, n_dv):
    # the first face of the top stays level, the faces after it rise
    c = cs.channel_case(8, 4, n_dv, sides={"top": {"kind": kind}}, U0=(40.0, 0.0, 0.0), flatten=False)
    p = np.array(c.mesh.points, dtype=np.float64)
    p[:, 1] *= 1.0 + 0.3 * np.maximum(p[:, 0] - 0.25, 0.0)
    c.mesh.points = p
    return c.flatten()


@pytest.mark.parametrize("precision", [dl.FP64, dl.FP32C])
@pytest.mark.parametrize("kind,n_dv", [("DVMsymmetry", 8), ("DVMsymmetry", 10), ("symmetryPlane", 8)])
def test_continued_run_is_the_run(kind, n_dv, precision):
    c = _tilted(kind, n_dv)
    a = dl.Solver(c, precision=precision)
    a.step(3, c.dt)
    b = dl.Solver(c, precision=precision)
    b.set_state(*a.state(), c.dt, a.step_record())
    for s in (a, b):
        s.step(2, c.dt)
    for x, y in zip(a.state(), b.state()):
        assert np.array_equal(x, y)
    ma, mb = a.macros(), b.macros()
    for k in ma:
        assert np.array_equal(ma[k], mb[k]), k

"""A state whose eddy viscosity is far below the floor (a field a user's program zeroed but for
round-off, say): the damping ratios are quotients of terms of the order CHI^2 and CHI, and both
are formed with one reciprocal of a product that must not underflow where they do not.  After
the first iteration the floor holds the field, so one iteration shows it.

Tolerance: that of the other FP64 parity tests, 1e-10 of each variable's maximum."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tnsgpu import cases
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("nu", [1e-30, 1e-100, 1e-112, 1e-125, 1e-150])
def test_one_iteration_from_a_vanishing_eddy_viscosity(nu, general):
    mesh, flow = cases.ramp_mesh(40, 20), cases.ramp_flow()
    if general:
        mesh, _ = cases.renumbered_mesh(mesh, seed=3)
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=5)
    c0[4] = c0[0] * nu
    ri = rinit_cold(flow)
    s = Solver(mesh, flow, ri)
    s.upload(c0)
    s.run(1, 0)  # raises where the state is not finite
    o = Oracle(mesh, flow, ri)
    o.set_state(c0)
    o.iterate(1, 1)
    got, ref = s.download(), o.state()
    s.close()
    assert np.all(np.isfinite(ref))
    err = np.max(np.abs(got - ref), axis=1) / np.max(np.abs(ref), axis=1)
    assert np.all(err < 1e-10), err

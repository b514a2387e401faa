"""The nu~ floor of the update, C5 = C1 max(RTOL, C5/C1), rounds the state: where it does not
bind, the quotient and the product should give back what the reference's division and
multiplication give.  A quotient formed with two roundings instead moved half of all cells by an
ulp, and C5's error against the oracle grew some thirtyfold.

Bound, from the scheme: one iteration changes C5 by 1e-2 of itself or less, with a relative
error near 1e-15 of that change, so 1e-17 of C5: that flips a rounding (an ulp, 1.1e-16 to
2.2e-16) in a few cells of a hundred, a mean of at most 4e-18 of the largest C5."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tnsgpu import cases
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,general", [
    (96, 32, False),    # one tile a block with extra thread rows
    (395, 255, False),  # without
    (1184, 96, False),  # the pipelined stage
    (96, 32, True),     # the general mesh's stage
])
def test_c5_rounds_as_the_reference_after_one_iteration(ni, nj, general):
    mesh, flow = cases.ramp_mesh(ni, nj), cases.ramp_flow()
    if general:
        mesh, _ = cases.renumbered_mesh(mesh, seed=3)
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=ni)
    c0[4] *= 30.0  # an eddy viscosity well above the floor
    ri = rinit_cold(flow)
    s = Solver(mesh, flow, ri)
    s.upload(c0)
    s.run(1, 0)
    o = Oracle(mesh, flow, ri)
    o.set_state(c0)
    o.iterate(1, 1)
    got, ref = s.download()[4], o.state()[4]
    s.close()
    assert np.mean(np.abs(got - ref)) <= 4e-18 * np.max(np.abs(ref))

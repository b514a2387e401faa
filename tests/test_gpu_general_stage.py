"""The general-mesh FP64 stage kernel (chunks of 256 cells, ghosts with their own face flux,
VIS gathered by stage 1) against the oracle: one chunk that is not full, exactly full, one cell
more, several chunks with ghosts of every type the families have, both time steps; and VIS as the
post-run query returns it.

Tolerance: that of the other FP64 parity tests, 1e-10 of each variable's maximum (the GPU
contracts a*b+c and uses its own transcendentals; three iterations differ by a few ulp of
the largest term).
"""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tnsgpu import cases
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("family,ni,nj,local", [
    ("ramp", 9, 7, 1),      # one short chunk
    ("plume", 16, 16, 1),   # one full chunk
    ("port", 257, 3, 1),    # three chunks and three cells; every cell of two rows has a ghost
    ("plume", 70, 41, 0),   # 11 chunks and a short one, global time step
    ("port", 64, 48, 1),    # type-6 ghosts across several chunks
])
def test_general_stage_matches_oracle(family, ni, nj, local):
    if family == "ramp":
        mesh, flow = cases.ramp_mesh(ni, nj), cases.ramp_flow()
    elif family == "plume":
        mesh, flow = cases.nozzle_plume_mesh(ni, nj), cases.nozzle_plume_flow()
    else:
        mesh, flow = cases.port_mesh(ni, nj), cases.port_flow()
    flow.local = local
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=ni + nj)
    ri = rinit_cold(flow)
    g, perm = cases.renumbered_mesh(mesh, seed=3)
    q0 = np.empty_like(c0)
    q0[:, perm] = c0
    s = Solver(g, flow, ri)
    s.upload(q0)
    rec = s.run(3, 3)
    o = Oracle(g, flow, ri)
    o.set_state(q0)
    ref_rec = o.iterate(3, 3)
    ref = o.state()
    err = np.max(np.abs(s.download() - ref), axis=1) / np.max(np.abs(ref), axis=1)
    assert np.all(err < TOL), err
    assert np.all(np.abs(rec - ref_rec) <= 1e-8 * np.abs(ref_rec)), (rec, ref_rec)
    s.close()

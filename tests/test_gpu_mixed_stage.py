"""The mixed-precision stage kernels at the edges of their block shapes: with the extra thread
rows of small meshes in both, one or no kernel, tiles and chunks cut short by the mesh's edge,
port ghosts, both time steps, axisymmetric and plane; bit for bit against the batched kernels.

Tolerance against the FP64 path: the state is FP64 and each iteration adds an increment formed
in FP32 from deviations, so three iterations differ by a few 2^-24 of what they change; the
bounds are those the mixed path is held to after fifty iterations (test_gpu_mixed), per variable
of its maximum.
"""
import numpy as np
import pytest

from tnsgpu import cases
from tnsgpu.batch import Batch
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu
TOL = np.array([2e-6, 1e-4, 1e-4, 2e-6, 5e-5])


def _case(family, ni, nj, local):
    if family == "ramp":
        mesh, flow = cases.ramp_mesh(ni, nj), cases.ramp_flow()
    elif family == "plume":
        mesh, flow = cases.nozzle_plume_mesh(ni, nj), cases.nozzle_plume_flow()
    else:
        mesh, flow = cases.port_mesh(ni, nj), cases.port_flow()
    flow.local = local
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=ni + nj)
    return mesh, flow, c0, rinit_cold(flow)


def _state(mesh, flow, ri, c0, precision, schedule=None):
    s = Solver(mesh, flow, ri, precision=precision)
    s.upload(c0)
    if schedule is None:
        s.run(3, 0)
    else:
        b = Batch([s], schedule=schedule)
        b.run(3, 0)
        b.close()
    q = s.download()
    s.close()
    return q


SIZES = [
    ("ramp", 9, 33, 1),      # a second tile one cell high and wide
    ("port", 60, 40, 1),     # extra rows in the stage and viscous kernels
    ("plume", 200, 250, 1),  # 200 tiles: in the stage kernel alone
    ("ramp", 395, 255, 0),   # 400 tiles: none, both edges partial, global time step
    ("plume", 290, 330, 1),  # the same, axisymmetric
]


@pytest.mark.parametrize("family,ni,nj,local", SIZES)
def test_mixed_follows_fp64_and_the_batch(family, ni, nj, local):
    mesh, flow, c0, ri = _case(family, ni, nj, local)
    ref = _state(mesh, flow, ri, c0, 0)
    q = _state(mesh, flow, ri, c0, 1)
    err = np.max(np.abs(q - ref), axis=1) / np.max(np.abs(ref), axis=1)
    assert np.all(err <= TOL), err
    for schedule in (0, 2):
        assert np.array_equal(q, _state(mesh, flow, ri, c0, 1, schedule))


@pytest.mark.parametrize("family,ni,nj,local", SIZES[:4])
def test_mixed_general_mesh_follows_fp64(family, ni, nj, local):
    mesh, flow, c0, ri = _case(family, ni, nj, local)
    g, perm = cases.renumbered_mesh(mesh, seed=5)
    q0 = np.empty_like(c0)
    q0[:, perm] = c0
    ref, q = (_state(g, flow, ri, q0, p) for p in (0, 1))
    err = np.max(np.abs(q - ref), axis=1) / np.max(np.abs(ref), axis=1)
    assert np.all(err <= TOL), err

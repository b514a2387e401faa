"""The pipelined stage kernel of large FP64 meshes (more tiles than resident blocks of the
one-tile-a-block kernel): against the oracle at sizes around its edges -- a last tile two
columns wide or one row high, a row length that is no multiple of 16 bytes (which takes the
other kernel), port sums, both time steps -- and bit for bit against the batched kernels,
which run a tile a block.

Tolerance: that of the other FP64 parity tests, 1e-10 of each variable's maximum (the GPU
contracts a*b+c and uses its own transcendentals; three iterations differ by a few ulp of
the largest term).
"""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tnsgpu import cases
from tnsgpu.batch import Batch
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu
TOL = 1e-10


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


@pytest.mark.parametrize("family,ni,nj,local", [
    ("ramp", 1200, 98, 1),    # last tile 2 columns wide
    ("ramp", 1185, 96, 0),    # last tile 1 row high, global time step
    ("plume", 1187, 110, 1),  # both edges partial, axisymmetric
    ("plume", 1200, 97, 1),   # odd rows: the other kernel
    ("port", 1192, 100, 1),   # type-6 ghosts in the halo
])
def test_large_mesh_matches_oracle(family, ni, nj, local):
    mesh, flow, c0, ri = _case(family, ni, nj, local)
    s = Solver(mesh, flow, ri)
    s.upload(c0)
    rec = s.run(3, 3)
    o = Oracle(mesh, flow, ri)
    o.set_state(c0)
    ref_rec = o.iterate(3, 3)
    ref = o.state()
    err = np.max(np.abs(s.download() - ref), axis=1) / np.max(np.abs(ref), axis=1)
    assert np.all(err < TOL), err
    assert np.all(np.abs(rec - ref_rec) <= 1e-8 * np.abs(ref_rec)), (rec, ref_rec)
    s.close()


def test_large_mesh_equals_batched_tiles_bitwise():
    mesh, flow, c0, ri = _case("plume", 1187, 110, 1)
    out = []
    for schedule in (None, 0, 3):
        s = Solver(mesh, flow, ri)
        s.upload(c0)
        if schedule is None:
            s.run(4, 2)
        else:
            b = Batch([s], schedule=schedule)
            b.run(4, 2)
            b.close()
        out.append(s.download())
        s.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("family,ni,nj,local", [
    ("plume", 200, 250, 1),  # 200 tiles: extra thread rows in the stage kernel alone
    ("ramp", 395, 255, 0),   # 400 tiles: none, odd rows, last tile short both ways
    ("port", 60, 40, 1),     # 16 tiles: extra rows in the stage and viscous kernels
])
def test_smaller_meshes_of_each_block_shape_match_oracle(family, ni, nj, local):
    test_large_mesh_matches_oracle(family, ni, nj, local)

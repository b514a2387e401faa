"""States of a mesh whose cells are numbered otherwise than the device's: what is uploaded is
downloaded again bit for bit, and is in the order the iterations expect -- one block of cells
with shuffled ids, and a general mesh; pageable and page-locked arrays; sizes below, at and above
a block of the renumbering kernel.  (No arithmetic: exact.)"""
import numpy as np
import pytest
import torch

from tnsgpu import cases
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj", [(5, 3), (16, 16), (257, 2), (67, 31)])
@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("locked", [False, True])
def test_state_round_trip_in_the_callers_numbering(ni, nj, rotate, precision, locked):
    flow = cases.ramp_flow()
    mesh = cases.ramp_mesh(ni, nj)
    g, perm = cases.renumbered_mesh(mesh, seed=2, rotate=rotate)
    c0, ri = cases.noisy_restart_state(flow, mesh.neles, seed=1)
    a = Solver(mesh, flow, ri, precision=precision)
    a.upload(c0)
    b = Solver(g, flow, ri, precision=precision)
    q = torch.empty((5, mesh.neles), dtype=torch.float64, pin_memory=locked).numpy()
    q[:, perm] = c0
    b.upload(q)
    out = torch.zeros((5, mesh.neles), dtype=torch.float64, pin_memory=locked).numpy()
    for arr in (b.download(), out):
        if arr is out:
            b._check(b.L.tns_download_state(b.h, *(out[k].ctypes.data for k in range(5))))
        assert np.array_equal(arr, q)
    if not rotate:  # one block: the same iterations as in its own order
        a.run(2, 0)
        b.run(2, 0)
        assert np.array_equal(b.download()[:, perm], a.download())
    a.close()
    b.close()

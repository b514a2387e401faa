"""The block shapes of the stage and viscous kernels in the builds with 4 and 16 rows a tile: blocks
with extra thread rows (few tiles), without, and the pipelined stage, on either side of each
rule's line on 148 SMs (296 tiles for the FP64 stage, 148 for the viscous kernels; 592 and 148 for
the mixed stage with 4 and 16 rows), against the oracle.

Tolerances: those of the other parity tests, 1e-10 of each variable's maximum in FP64, in mixed
precision (2e-6, 1e-4, 1e-4, 2e-6, 5e-5)."""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tnsgpu import _lib, cases
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ti,ni,nj", [
    (16, 257, 255),  # 136 tiles
    (16, 330, 255),  # 168
    (16, 400, 254),  # 200, and rows the pipelined stage can address
    (4, 144, 255),   # 288
    (4, 290, 255),   # 584
    (4, 300, 255),   # 600
    (4, 500, 254),   # 1000, the pipelined stage
])
def test_block_shapes_match_the_oracle(ti, ni, nj, precision):
    mesh, flow = cases.ramp_mesh(ni, nj), cases.ramp_flow()
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=ni)
    ri = rinit_cold(flow)
    s = Solver(mesh, flow, ri, precision=precision, lib=_lib.variant_path(ti))
    s.upload(c0)
    s.run(3, 3)
    o = Oracle(mesh, flow, ri)
    o.set_state(c0)
    o.iterate(3, 3)
    ref = o.state()
    err = np.max(np.abs(s.download() - ref), axis=1) / np.max(np.abs(ref), axis=1)
    s.close()
    assert np.all(err < (np.array([2e-6, 1e-4, 1e-4, 2e-6, 5e-5]) if precision else 1e-10)), err

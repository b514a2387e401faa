"""The persistent kernel of mixed batches (schedule 3) at both of its register budgets and with
its pre-passes in pairs and apart: the states of every case, active or masked, equal those of
the case run alone bit for bit (the same tile functions in the same order of operations).

Tiles of 8 x 32 cells on 148 SMs: up to 444 tiles the kernel with three blocks an SM, to 592 the
one with four, to 888 three again (two rounds either way), then four; pairs from 444 or 592 on."""
import numpy as np
import pytest

from tnsgpu import cases
from tnsgpu.batch import Batch
from tnsgpu.formats import rinit_cold
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu


def _solver(ni, nj, seed):
    mesh, flow = cases.ramp_mesh(ni, nj), cases.ramp_flow()
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=seed)
    s = Solver(mesh, flow, rinit_cold(flow), precision=1)
    s.upload(c0)
    return s


@pytest.mark.parametrize("sizes", [
    [(33, 31), (41, 70)],                # 23 tiles, edges short
    [(512, 192), (200, 65)],             # 459: four blocks an SM, fewer tiles than blocks
    [(512, 192), (512, 128), (96, 32)],  # 652: three, more tiles than blocks
    [(512, 192), (512, 192), (400, 127)],  # 968: four, more tiles than blocks
], ids=["23", "459", "652", "968"])
@pytest.mark.parametrize("masked", [False, True], ids=["all", "masked"])
def test_persistent_mixed_batch_equals_solo_runs(sizes, masked):
    batch = [_solver(ni, nj, k) for k, (ni, nj) in enumerate(sizes)]
    solo = [_solver(ni, nj, k) for k, (ni, nj) in enumerate(sizes)]
    b = Batch(batch, schedule=3)
    b.run(5, 0)
    for s in solo:
        s.run(5, 0)
    if masked:  # the last case rests
        b.set_active([k < len(sizes) - 1 for k in range(len(sizes))])
        b.run(3, 0)
        for s in solo[:-1]:
            s.run(3, 0)
    for a, s in zip(batch, solo):
        assert np.array_equal(a.download(), s.download())
    b.close()
    for s in batch + solo:
        s.close()

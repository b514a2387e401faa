"""The recorded iteration of the adjoint on meshes large enough for the pipelined stage (more than
444 tiles on 148 SMs, rows of even length), whose tensor maps then name the caller's own arrays:
with arrays aligned to 16 bytes, which take it, and to 8 bytes only, which TMA cannot address and
which must take the other kernel.  Both give the solver's own iteration and the same record bit
for bit, and the reverse of each agrees with autograd.

Tolerances: bit equality for the states and records (the same arithmetic per cell); 1e-10 of each
component's maximum for lambda, as in the other comparisons of a reverse step with autograd."""
import numpy as np
import pytest
import torch

from oracle.adjoint_restatement import RestatedScheme
from tnsgpu import cases, formats
from tnsgpu.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,ni,nj,local", [
    ("ramp", 1200, 98, 1),  # 600 tiles, the last two columns wide
    ("ramp", 1186, 96, 0),  # 447, the last two rows high, global time step
    ("port", 1192, 100, 1),  # type-6 ghosts
])
def test_recorded_step_through_the_pipelined_stage(family, ni, nj, local):
    mesh, flow = (cases.ramp_mesh(ni, nj), cases.ramp_flow()) if family == "ramp" else \
        (cases.port_mesh(ni, nj), cases.port_flow())
    flow.local = local
    ri = formats.rinit_cold(flow)
    c0, _ = cases.noisy_restart_state(flow, mesh.neles, seed=ni)
    n = mesh.neles
    solo = Solver(mesh, flow, ri)
    solo.upload(c0)
    solo.run(1, 0)
    own = solo.download()
    solo.close()
    lam0 = np.random.default_rng(1).normal(size=(5, n))
    s = Solver(mesh, flow, ri)
    rec_size = s.adjoint_record_size()

    def run(off):
        """Arrays that start `off` doubles into their allocations."""
        def array(size):
            a = torch.zeros(size + 2, device="cuda", dtype=torch.float64)[off:off + size]
            assert a.data_ptr() % 16 == (0 if off % 2 == 0 else 8)
            return a
        q, qn, rec, lam = array(5 * n), array(5 * n), array(rec_size), array(5 * n)
        q.copy_(torch.tensor(c0.reshape(-1)))
        lam.copy_(torch.tensor(lam0.reshape(-1)))
        torch.cuda.synchronize()
        s.adjoint_record(q.data_ptr(), qn.data_ptr(), rec.data_ptr())
        s.adjoint_step(q.data_ptr(), lam.data_ptr(), False, rec_ptr=rec.data_ptr())
        torch.cuda.synchronize()
        return qn.cpu().numpy().reshape(5, n), rec.cpu().numpy(), lam.cpu().numpy().reshape(5, n)

    (qa, ra, la), (qb, rb, lb) = run(0), run(1)
    s.close()
    assert np.array_equal(qa, own) and np.array_equal(qb, own)
    assert np.array_equal(ra, rb)
    sch = RestatedScheme(mesh, flow, device="cuda", rinit=ri)
    Q = torch.tensor(c0.reshape(5, ni, nj), device="cuda", requires_grad=True)
    G = sch.iteration(Q, sch.geometry(sch.x0, sch.y0), sch.params())
    (ref,) = torch.autograd.grad(G, [Q], grad_outputs=torch.tensor(lam0.reshape(5, ni, nj), device="cuda"))
    ref = ref.cpu().numpy().reshape(5, n)
    for got in (la, lb):
        assert np.all(np.max(np.abs(got - ref), axis=1) < 1e-10 * np.max(np.abs(ref), axis=1))

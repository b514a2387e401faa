"""The reverse of a global time step (LOCAL = 0): DTMIN's adjoint goes to the cell whose step
DTMIN is, which the kernel finds by comparing that cell's step with DTMIN bit for bit.  Where
the two round differently no cell is found and the whole term is missing, up to a tenth of
lambda's maximum.

Tolerances: those of the other comparisons of a CUDA reverse step with autograd, 1e-10 of
each component's maximum of lambda and 1e-9 of a parameter's gradient."""
import numpy as np
import pytest
import torch

from oracle.adjoint_restatement import RestatedScheme
from tnsgpu import adjoint, cases, formats

pytestmark = pytest.mark.gpu
FAMILIES = {
    "ramp": (lambda: cases.ramp_mesh(40, 16), cases.ramp_flow),
    "nozzle2d": (lambda: cases.nozzle_2d_mesh(36, 18), cases.nozzle_2d_flow),
    "plume": (lambda: cases.nozzle_plume_mesh(48, 20), cases.nozzle_plume_flow),
}


def _scheme(family):
    mesh, base = FAMILIES[family][0](), FAMILIES[family][1]()
    flow = formats.Flow(**{**base.__dict__, "local": 0})
    return mesh, flow, RestatedScheme(mesh, flow, device="cuda", rinit=formats.rinit_cold(flow))


def _compare(mesh, flow, sch, C, lam):
    """One reverse step on the device against autograd: lambda and the parameter gradients."""
    space = adjoint.DesignSpace(sch)
    params, _ = adjoint._leaves(sch, None, None, None, None)
    prm = adjoint.Params(params[0], params[1], params[2], flow)
    Q = C.clone().requires_grad_(True)
    G = sch.iteration(Q, sch.geometry(sch.x0, sch.y0), prm)
    ref = torch.autograd.grad(G, [Q] + params, grad_outputs=lam, allow_unused=True)
    dev = adjoint.DeviceAdjoint(sch, space, prm, None)
    try:
        got = lam.clone().contiguous()
        dev.step(C.contiguous(), got, True)
        sens = dev.sensitivities()
    finally:
        dev.close()
    err = torch.amax(torch.abs(got - ref[0]), dim=(1, 2)) / torch.amax(torch.abs(ref[0]), dim=(1, 2))
    assert float(err.max()) < 1e-10, err
    gp = adjoint._parameter_gradient(sch, space, params, None, sens, None)
    for k in range(3):
        r = float(ref[k + 1]) if ref[k + 1] is not None else 0.0
        assert abs(float(gp[k]) - r) <= 1e-9 * max(abs(r), 1e-300), (k, float(gp[k]), r)


@pytest.mark.parametrize("family", sorted(FAMILIES))
@pytest.mark.parametrize("seed", range(6))
def test_global_time_step_reverse_on_many_states(family, seed):
    mesh, flow, sch = _scheme(family)
    rng = np.random.default_rng(100 + seed)
    c0 = formats.cold_state(flow, mesh.neles, formats.rinit_cold(flow))
    c0 = c0 * (1 + 2e-2 * rng.uniform(-1, 1, c0.shape))
    c0[2] = 0.05 * c0[1] * rng.uniform(-1, 1, mesh.neles)
    C = torch.tensor(c0.reshape(5, *mesh.shape), device="cuda")
    prm0, geo0 = sch.params(), sch.geometry(sch.x0, sch.y0)
    with torch.no_grad():
        for _ in range(10):
            C = sch.iteration(C, geo0, prm0)
    lam = torch.tensor(rng.normal(size=(5,) + mesh.shape), device="cuda")
    _compare(mesh, flow, sch, C, lam)


def test_global_time_step_reverse_where_cells_share_the_minimum():
    """A uniform state on a flat wall: every cell of the first row has the same step, and each
    gets an equal part of DTMIN's adjoint."""
    mesh, base = cases.ramp_mesh(40, 16, 0.0), cases.ramp_flow()
    flow = formats.Flow(**{**base.__dict__, "local": 0})
    sch = RestatedScheme(mesh, flow, device="cuda", rinit=formats.rinit_cold(flow))
    c0 = formats.cold_state(flow, mesh.neles, formats.rinit_cold(flow))
    C = torch.tensor(c0.reshape(5, *mesh.shape), device="cuda")
    lam = torch.tensor(np.random.default_rng(7).normal(size=(5,) + mesh.shape), device="cuda")
    _compare(mesh, flow, sch, C, lam)

"""The allocation-free time step at the sizes where its route changes (one cluster of eight blocks
up to 32768 cells, a grid with scratch beyond) and at the edges of threads, blocks and rounds:
DT of every cell against the formula in numpy, and DTMIN the smallest of the DT it wrote, bit
for bit (a minimum rounds nothing); each size twice, since the grid's counter is left for the
next call.

Tolerance of DT: eight roundings of relative size 1.1e-16, the subtraction of the kinetic energy
(at most a tenth of the energy here) amplifying two of them a little: 1e-15."""
import ctypes as C

import numpy as np
import pytest
import torch

from tnsgpu import _lib, cases, formats
from tnsgpu.solver import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 2047, 2048, 2049, 8193, 32767, 32768, 32769, 33793, 100001])
def test_dt_and_its_minimum(n):
    flow = cases.ramp_flow()
    params = make_params(flow, formats.rinit_cold(flow))
    rng = np.random.default_rng(n)
    base = formats.cold_state(flow, 1)[:, 0]
    rho = base[0] * (1 + 0.1 * rng.uniform(-1, 1, n))
    u, v = 200 * rng.uniform(-1, 1, n), 100 * rng.uniform(-1, 1, n)
    e = base[3] / base[0] * (1 + 0.01 * rng.uniform(-1, 1, n)) + 0.5 * (u * u + v * v)
    q = np.stack([rho, rho * u, rho * v, rho * e, rho * 1e-5])
    cfldl = flow.cfl * 10 ** rng.uniform(-5, -3, n)
    rr = 8314.0 / flow.amol
    u, v = q[1] / q[0], q[2] / q[0]
    t = (q[3] / q[0] - 0.5 * (u * u + v * v)) / (rr / (flow.gama - 1.0))
    ref = cfldl / (np.sqrt(u * u + v * v) + np.sqrt(flow.gama * rr * t))
    dq, dc = torch.tensor(q, device="cuda"), torch.tensor(cfldl, device="cuda")
    for _ in range(2):
        dt = torch.full((n + 1,), -1.0, device="cuda", dtype=torch.float64)
        dtmin = torch.full((2,), -1.0, device="cuda", dtype=torch.float64)
        rc = _lib.load().tns_time_step_noalloc(dq.data_ptr(), dc.data_ptr(), n, C.byref(params), dt.data_ptr(),
                                               dtmin.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        got = dt.cpu().numpy()
        assert got[n] == -1.0 and float(dtmin[1]) == -1.0
        assert np.max(np.abs(got[:n] - ref) / ref) < 1e-15
        assert float(dtmin[0]) == got[:n].min()

"""Navier-Stokes at an infinite Reynolds number (viscosity exactly zero, no artificial dissipation): the time derivative is
the Euler build's, on single-order and mixed-order meshes, and a state that has turned to NaN leaves nothing behind for
the next one."""
import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases
from cases_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(hg.PREC_FP64, 1e-12), (hg.PREC_FP32, 1e-4)])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("viscous", [hg.BR1, hg.IP])
def test_infinite_reynolds_number(viscous, mixed, precision, tol):
    N = np.where(np.isin(np.arange(72) % 9, (3, 4, 5)), 5, 4) if mixed else 4
    d = hmesh.box_descriptor(9, 8, 0.0, 1.0, 0.0, 1.0, N, hg.NODES_LG)
    kw = dict(mach=0.3, node_type=hg.NODES_LG, riemann=hg.ROE, precision=precision, bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    x = d["x"].reshape(-1, 2)
    Q = cases.kelvin_helmholtz(x[:, 0], x[:, 1], seed=2).ravel()
    e = hg.GpuDGSEM(d, **kw)
    e.set_state(Q)
    ref = e.compute_time_derivative(0.0)
    g = hg.GpuDGSEM(d, navier_stokes=1, reynolds=np.inf, viscous=viscous, ip_method=hg.SIPG, sigma0_ip=5.0, **kw)
    g.set_state(np.full_like(Q, np.nan))
    for k in range(2):   # both parities of the trace buffers
        try:
            g.time_step(hg.SCHEME_RK3, 0.0, 1e-6)
        except hg.HorsesGpuError:
            pass
    g.set_state(Q)
    assert rel_l2(g.compute_time_derivative(0.0), ref) <= tol
    g.time_steps(hg.SCHEME_RK3, 2, 0.0, 1e-6)
    e.time_steps(hg.SCHEME_RK3, 2, 0.0, 1e-6)
    assert rel_l2(g.state(), e.state()) <= tol

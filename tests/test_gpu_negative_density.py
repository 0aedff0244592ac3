"""A node of negative density whose element's traces are still positive (an undershoot at an interior Gauss node): the
fluxes stay finite in both precisions, as 1 / rho does, so the time derivative is the oracle's and the default health
policy records the density and steps on."""
import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases
from oracle import oracle as O
from cases_util import perturbed, rel_l2

N, P = 4, 5


def problem(ns):
    m = hmesh.cartesian(3, 3, 0.0, 1.0, 0.0, 1.0)
    kw = dict(nodes=O.LG, riemann=O.ROE, mach=0.3)
    if ns:
        kw.update(reynolds=200.0, navier_stokes=1, viscous=O.BR1)
    orc = O.Oracle(m, N, bcs=hmesh.periodic_bcs_cartesian(), **kw)
    X = orc.coords()
    Q = perturbed(cases.kelvin_helmholtz(X[:, 0], X[:, 1], seed=3).ravel(), 0.02, seed=4).reshape(9, P, P, 4)
    Q[4, 2, 2, 0] = -0.05
    return orc, kw, Q.ravel()


def test_traces_of_the_case_are_positive():
    Q = problem(False)[2].reshape(9, P, P, 4)
    xi, _ = np.polynomial.legendre.leggauss(P)
    V = np.polynomial.legendre.legvander(xi, N)
    lb = np.polynomial.legendre.legvander(np.array([-1.0, 1.0]), N) @ np.linalg.inv(V)
    assert Q[4, 2, 2, 0] < 0.0
    for tr in (np.einsum("bj,ejik->ebik", lb, Q), np.einsum("bi,ejik->ebjk", lb, Q)):
        p = 0.4 * (tr[..., 3] - 0.5 * (tr[..., 1] ** 2 + tr[..., 2] ** 2) / tr[..., 0])
        assert tr[..., 0].min() > 0.0 and p.min() > 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(hg.PREC_FP64, 1e-12), (hg.PREC_FP32, 1e-4)])
@pytest.mark.parametrize("ns", [False, True])
def test_negative_density_at_an_interior_node(ns, precision, tol):
    orc, kw, Q = problem(ns)
    kw = {k: v for k, v in kw.items() if k != "nodes"}
    g = hg.GpuDGSEM(orc.export_mesh(), precision=precision, node_type=O.LG, bcs=[dict(type=hg.BC_PERIODIC)] * 4, **kw)
    orc.set_state(Q)
    ref = orc.time_derivative(0.0)
    assert np.isfinite(ref).all()
    g.set_state(Q)
    assert rel_l2(g.compute_time_derivative(0.0), ref) <= tol
    for k in range(2):
        g.time_step(hg.SCHEME_EULER, 0.0, 1e-9)
    g.synchronize()
    assert g.health() == (hg.HEALTH_DENSITY | g.health()[0] & hg.HEALTH_PRESSURE, 4)

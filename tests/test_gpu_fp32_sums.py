"""Time derivatives in 32 bits keep the digits of their fixture (golden/fp32_sums.npz, the output of the kernels that held
one node per thread): a node's sums are taken in one order.  The vortex is smooth, so its time derivative is a
difference of sums a thousand times as large and another order changes it by 5e-5 and more in the 2-norm; the residual
maxima of the cylinder's impulsive start change by 1e-6 to 5e-5.  Bound: 16 units in the last place of 32 bits, for the
last bits of single terms."""
import os

import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases
from cases_util import GOLDEN, rel_l2

TOL = 16 * 2.0 ** -24
EULER = [(N, nodes, riemann) for N, nodes in ((1, hg.NODES_LG), (2, hg.NODES_LGL), (4, hg.NODES_LGL), (5, hg.NODES_LG), (8, hg.NODES_LG))
         for riemann in (hg.ROE, hg.HLL, hg.LXF)]
CYLINDER = [(9, 27, 5), (15, 40, 2), (12, 32, 3), (12, 60, 6)]


def euler_context(N, nodes, riemann):
    d = hmesh.box_descriptor(9, 5, -5.0, 5.0, -5.0, 5.0, N, nodes)
    x = d["x"].reshape(-1, 2)
    g = hg.GpuDGSEM(d, mach=0.5, node_type=nodes, riemann=riemann, precision=hg.PREC_FP32, bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    return g, cases.isentropic_vortex(x[:, 0], x[:, 1], mach=0.5, beta=4.0, xc=0.3, yc=-0.2).ravel()


def cylinder_context(nr, nt, N, seed):
    u = np.sqrt(1.4) * 0.2
    stream = np.array([1.0, u, 0.0, 2.5 + 0.5 * u * u])
    d = hmesh.build_descriptor(hmesh.ogrid(nr, nt, 0.5, 30.0, 1.05), N, hg.NODES_LG)
    g = hg.GpuDGSEM(d, mach=0.2, reynolds=100.0, prandtl=0.72, navier_stokes=1, viscous=hg.BR1, node_type=hg.NODES_LG,
                    riemann=hg.ROE, precision=hg.PREC_FP32, bcs=[dict(type=hg.BC_VISCOUSWALL, wall_type=2),
                                                                 dict(type=hg.BC_FARFIELD, state=stream)])
    n = len(d["jac"])
    return g, np.tile(stream, n) + 1e-3 * np.random.default_rng(seed).standard_normal(4 * n)


def euler_derivative(N, nodes, riemann, variant):
    g, Q = euler_context(N, nodes, riemann)
    g.set_tiling(variant)
    g.set_state(Q)
    return g.compute_time_derivative(0.0)


def cylinder_residuals(nr, nt, N):
    out = []
    for seed in range(4):
        g, Q = cylinder_context(nr, nt, N, seed)
        g.set_state(Q)
        g.compute_time_derivative(0.0)
        out.append(g.residuals())
        g.time_step(hg.SCHEME_RK3, 0.0, 1e-6)
        out.append(g.residuals())
    return np.array(out)


@pytest.fixture(scope="module")
def golden():
    return np.load(os.path.join(GOLDEN, "fp32_sums.npz"))


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("N,nodes,riemann", EULER)
def test_euler_time_derivative(golden, N, nodes, riemann, variant):
    assert rel_l2(euler_derivative(N, nodes, riemann, variant), golden["euler_%d_%d_%d" % (N, nodes, riemann)]) <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("nr,nt,N", CYLINDER)
def test_cylinder_residual_maxima(golden, nr, nt, N):
    r, ref = cylinder_residuals(nr, nt, N), golden["cylinder_%d_%d_%d" % (nr, nt, N)]
    assert all(rel_l2(a, b) <= TOL for a, b in zip(r, ref))

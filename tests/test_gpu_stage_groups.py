"""The Euler stage kernel's element groups: orders at both ends of every group-size rule, meshes whose last
group is partly empty, meshes with more groups than resident CTAs (a CTA then walks over several groups with
its prefetch running), against the oracle (residual: relative L2 <= 1e-12 in FP64, 1e-4 in FP32, the suite's
bounds), and the traces a stage leaves against those formed from the same state by hg_set_state (bitwise)."""
import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases
from oracle import oracle as O
from cases_util import perturbed, rel_l2

pytestmark = pytest.mark.gpu


def box(nx, ny, N, nodes, precision=hg.PREC_FP64):
    m = hmesh.cartesian(nx, ny, -5.0, 5.0, -5.0, 5.0)
    orc = O.Oracle(m, N, nodes=nodes, riemann=O.ROE, mach=0.5, bcs=hmesh.periodic_bcs_cartesian())
    X = orc.coords()
    Q = perturbed(cases.isentropic_vortex(X[:, 0], X[:, 1]).ravel(), 0.02, seed=N)
    g = hg.GpuDGSEM(orc.export_mesh(), mach=0.5, node_type=nodes, riemann=hg.ROE, precision=precision,
                    bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    return orc, g, Q


@pytest.mark.parametrize("nx,ny,N,nodes", [
    (1, 1, 4, O.LGL), (3, 1, 1, O.LG), (5, 7, 2, O.LG), (5, 7, 4, O.LG), (5, 7, 5, O.LGL), (3, 5, 7, O.LG),
    (3, 5, 8, O.LG), (3, 3, 9, O.LGL), (3, 3, 10, O.LG), (2, 3, 12, O.LG),
    (171, 163, 1, O.LG), (171, 163, 1, O.LGL), (97, 61, 4, O.LGL), (97, 61, 4, O.LG), (53, 47, 6, O.LG), (61, 41, 8, O.LG)])
@pytest.mark.parametrize("precision", [hg.PREC_FP64, hg.PREC_FP32])
def test_groups_against_oracle(nx, ny, N, nodes, precision):
    orc, g, Q = box(nx, ny, N, nodes, precision)
    tol = 1e-12 if precision == hg.PREC_FP64 else 1e-4
    orc.set_state(Q)
    ref = orc.time_derivative(0.0)
    dt = orc.estimate_dt(0.1, 1.0)
    for k in range(2):
        orc.time_step(O.RK3, k * dt, dt)
    for v in range(hg.lib.TILINGS):
        g.set_tiling(v)
        g.set_state(Q)
        assert rel_l2(g.compute_time_derivative(0.0), ref) <= tol
        assert np.allclose(g.residuals(), np.abs(ref.reshape(-1, 4)).max(0), rtol=100 * tol)
        g.time_steps(hg.SCHEME_RK3, 2, 0.0, dt)
        assert rel_l2(g.state(), orc.state()) <= tol


@pytest.mark.parametrize("N", [1, 3, 4, 6, 7, 10])
def test_stage_traces_equal_those_of_a_loaded_state(N):
    orc, g, Q = box(9, 5, N, O.LG)
    _, h, _ = box(9, 5, N, O.LG)
    orc.set_state(Q)
    dt = orc.estimate_dt(0.1, 1.0)
    g.set_state(Q)
    g.time_steps(hg.SCHEME_RK3, 3, 0.0, dt)
    h.set_state(g.state())
    g.time_steps(hg.SCHEME_RK3, 2, 0.0, dt)
    h.time_steps(hg.SCHEME_RK3, 2, 0.0, dt)
    assert np.array_equal(g.state(), h.state())

"""The Navier-Stokes kernels' element groups: orders at both ends of every group-size rule, meshes whose last
group is partly empty, meshes with more groups than resident CTAs, with and without element-local gradients in a
group (artificial viscosity on some elements only), against the oracle (residual and RK3 steps: relative L2
<= 1e-12 in FP64, 1e-4 in FP32, the suite's bounds); and a context whose state is loaded against one that stepped
there (bitwise where the traces are the only thing carried over)."""
import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases
from oracle import oracle as O
from cases_util import perturbed, rel_l2

pytestmark = pytest.mark.gpu


def box(nx, ny, N, viscous, av, precision, nodes=O.LG, reynolds=200.0):
    m = hmesh.cartesian(nx, ny, 0.0, 1.0, 0.0, 1.0)
    okw = dict(nodes=nodes, riemann=O.ROE, mach=0.3, reynolds=reynolds, navier_stokes=1, viscous=viscous, ip_method=0,
               sigma0_ip=5.0)
    if av:
        okw.update(av_type=O.AV_LAPLACIAN, av_intensity=1.0)
    orc = O.Oracle(m, N, bcs=hmesh.periodic_bcs_cartesian(), av_indicator=O.IND_MODAL if av else 0, **okw)
    X = orc.coords()
    Q = cases.kelvin_helmholtz(X[:, 0], X[:, 1], delta=0.05, eps=0.05, seed=N, drho=1.0).ravel()
    # noise on a third of the elements only: the modal indicator flags some of them
    e = np.arange(nx * ny) % 3 == 0
    mask = np.repeat(e, 4 * (N + 1) ** 2)
    Q = np.where(mask, perturbed(Q, 0.02, seed=N), Q)
    kw = {k: v for k, v in okw.items() if k != "nodes"}
    g = hg.GpuDGSEM(orc.export_mesh(), precision=precision, node_type=nodes, bcs=[dict(type=hg.BC_PERIODIC)] * 4, **kw)
    if av:
        g.set_sensor(hg.SENSOR_MODAL)
    return orc, g, Q


@pytest.mark.parametrize("nx,ny,N,viscous,av", [
    (3, 3, 1, O.IP, False), (5, 7, 2, O.BR1, True), (5, 7, 3, O.IP, True), (5, 3, 4, O.BR1, False), (5, 3, 5, O.IP, True),
    (3, 5, 6, O.BR1, True), (3, 3, 7, O.IP, True), (3, 3, 8, O.IP, False), (3, 3, 9, O.BR1, False), (3, 3, 10, O.IP, True),
    (97, 61, 3, O.IP, True), (61, 41, 4, O.BR1, False), (53, 47, 5, O.IP, True), (41, 35, 7, O.IP, True),
    (41, 35, 7, O.BR1, True), (31, 29, 8, O.IP, False)])
@pytest.mark.parametrize("precision", [hg.PREC_FP64, hg.PREC_FP32])
def test_groups_against_oracle(nx, ny, N, viscous, av, precision):
    orc, g, Q = box(nx, ny, N, viscous, av, precision)
    tol = 1e-12 if precision == hg.PREC_FP64 else 1e-4
    orc.set_state(Q)
    ref = orc.time_derivative(0.0)
    dt = 1e-3 / (max(nx, ny) * (N + 1)) ** 2
    for k in range(2):
        orc.time_step(O.RK3, k * dt, dt)
    for v in range(hg.lib.TILINGS):
        g.set_tiling(v)
        g.set_state(Q)
        assert rel_l2(g.compute_time_derivative(0.0), ref) <= tol
        assert np.allclose(g.residuals(), np.abs(ref.reshape(-1, 4)).max(0), rtol=100 * tol)
        g.time_steps(hg.SCHEME_RK3, 2, 0.0, dt)
        assert rel_l2(g.state(), orc.state()) <= tol


@pytest.mark.parametrize("precision", [hg.PREC_FP64, hg.PREC_FP32])
@pytest.mark.parametrize("N", [2, 5, 7])
def test_stepped_and_loaded_states_agree(N, precision):
    """Inviscid interior penalty with the modal indicator: traces and indicator carried from the stage kernel or
    formed from the loaded state are the same bits."""
    orc, g, Q = box(9, 7, N, O.IP, True, precision, reynolds=0.0)
    _, h, _ = box(9, 7, N, O.IP, True, precision, reynolds=0.0)
    dt = 1e-3 / (9 * (N + 1)) ** 2
    g.set_state(Q)
    g.time_steps(hg.SCHEME_RK3, 3, 0.0, dt)
    h.set_state(g.state())
    g.time_steps(hg.SCHEME_RK3, 2, 0.0, dt)
    h.time_steps(hg.SCHEME_RK3, 2, 0.0, dt)
    assert np.array_equal(g.state(), h.state())


def test_sensor_kinds_take_turns_in_one_process():
    """Learned, modal, learned contexts of one order and precision: the learned ones launch the same kernels with the
    network's weights in shared memory, whatever ran in between."""
    from test_gpu_sensor import random_problem
    p, _, _, _ = random_problem(1, 7)
    states = []
    for kind in (hg.SENSOR_LEARNED, hg.SENSOR_MODAL, hg.SENSOR_LEARNED):
        for viscous in (O.IP, O.BR1):
            orc, g, Q = box(9, 7, 3, viscous, True, hg.PREC_FP32)
            if kind == hg.SENSOR_LEARNED:
                g.set_sensor(kind, mlp=p)
            g.set_state(Q)
            g.time_steps(hg.SCHEME_RK3, 2, 0.0, 1e-7)
            states.append(g.state())
    assert all(np.isfinite(s).all() for s in states)
    assert np.array_equal(states[0], states[4]) and np.array_equal(states[1], states[5])

"""hg_residuals reduces the partials of the last launch that wrote them, whichever way it was launched.  With the learned
sensor a step's last stage has the network's weights in shared memory and fewer CTAs than a bare time derivative; a
derivative between two replayed steps (or pairs of steps, or group steps) must not leave its partials to the second
one.  The derivative in between is of a rough state, whose residual is larger everywhere; the twin context runs plain
launches (timing mode), so both give the same bits."""
import numpy as np
import pytest
import torch

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases

pytestmark = pytest.mark.gpu

SIZES = [(3, 512, 64, hg.PREC_FP32), (7, 96, 64, hg.PREC_FP32), (7, 96, 64, hg.PREC_FP64)]


def network():
    r = np.random.default_rng(3)
    return r.normal(0.0, 0.2, hg.lib.MLP_PARAMS).astype(np.float32)


def context(N, nx, ny, precision, learned=True):
    d = hmesh.box_descriptor(nx, ny, 0.0, 1.0, 0.0, 1.0, N, hg.NODES_LG)
    g = hg.GpuDGSEM(d, mach=0.3, reynolds=1.0e3, navier_stokes=1, viscous=hg.IP, ip_method=hg.SIPG, sigma0_ip=5.0,
                    node_type=hg.NODES_LG, riemann=hg.ROE, av_type=hg.AV_LAPLACIAN, av_intensity=1.0, precision=precision,
                    bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    if learned:
        g.set_sensor(hg.SENSOR_LEARNED, mlp=network())
    x = d["x"].reshape(-1, 2)
    Q = cases.kelvin_helmholtz(x[:, 0], x[:, 1], delta=0.05, eps=0.05, seed=N, drho=1.0).ravel()
    rough = Q * (1.0 + 0.05 * np.random.default_rng(N).standard_normal(Q.shape))
    return g, Q, rough


@pytest.mark.parametrize("N,nx,ny,precision", SIZES)
def test_single_steps_around_a_time_derivative(N, nx, ny, precision):
    (a, Q, rough), (b, _, _) = context(N, nx, ny, precision), context(N, nx, ny, precision)
    b.profile(True)
    res, dt = [], 1e-8
    for g in (a, b):
        g.set_state(Q)
        for k in range(4):   # a graph per trace parity: plain, plain, captured, captured
            g.time_step(hg.SCHEME_RK3, k * dt, dt)
        g.set_state(rough)
        g.compute_time_derivative(0.0)
        big = g.residuals()
        g.set_state(Q)
        g.time_step(hg.SCHEME_RK3, 0.0, dt)
        res.append(g.residuals())
        assert (big > res[-1]).all()
    np.testing.assert_array_equal(res[0], res[1])


@pytest.mark.parametrize("N,nx,ny,precision", SIZES)
def test_step_pairs_around_a_time_derivative(N, nx, ny, precision):
    (a, Q, rough), (b, _, _) = context(N, nx, ny, precision), context(N, nx, ny, precision)
    b.profile(True)
    res, dt = [], 1e-8
    for g in (a, b):
        g.set_state(Q)
        g.time_step(hg.SCHEME_RK3, 0.0, dt)
        g.time_steps(hg.SCHEME_RK3, 7, 0.0, dt)   # one step, then a graph of two at the parity of a loaded state
        g.set_state(rough)
        g.compute_time_derivative(0.0)
        g.set_state(Q)
        g.time_steps(hg.SCHEME_RK3, 6, 0.0, dt)
        res.append(g.residuals())
    np.testing.assert_array_equal(res[0], res[1])


def test_group_steps_around_a_time_derivative():
    N, nx, ny, precision = SIZES[1]
    stream = torch.cuda.Stream()
    res, dt = [], 1e-8
    for grouped in (True, False):
        ms = [context(N, nx, ny, precision), context(5, 24, 24, precision)]
        gs = [m[0] for m in ms]
        for g, Q, _ in ms:
            g.set_stream(stream.cuda_stream)
            g.set_state(Q)
        group = hg.GpuGroup(gs) if grouped else None

        def steps(n):
            if grouped:
                group.time_steps(hg.SCHEME_RK3, n, 0.0, dt)
            else:
                for g in gs:
                    for k in range(n):
                        g.time_step(hg.SCHEME_RK3, 0.0, dt)
        if not grouped:
            for g in gs:
                g.profile(True)
        steps(1)
        steps(7)
        for g, _, rough in ms:
            g.set_state(rough)
            g.compute_time_derivative(0.0)
        for g, Q, _ in ms:
            g.set_state(Q)
        steps(6)
        res.append(np.array([g.residuals() for g in gs]))
    np.testing.assert_array_equal(res[0], res[1])

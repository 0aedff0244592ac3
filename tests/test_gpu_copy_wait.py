"""A stage kernel whose copies do not land in time: with a poll limit of 0 every wait gives up at once, the CTAs leave
before they read anything the copies bring, and the calls fail (status 1, HEALTH_COPY) until a new state is set."""
import ctypes as C

import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases

pytestmark = pytest.mark.gpu


def context(kind, precision):
    mixed = kind == "mixed"
    N = np.where(np.isin(np.arange(72) % 9, (3, 4, 5)), 5, 4) if mixed else 4
    d = hmesh.box_descriptor(9, 8, 0.0, 1.0, 0.0, 1.0, N, hg.NODES_LG)
    kw = dict(mach=0.3, node_type=hg.NODES_LG, riemann=hg.ROE, bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    if kind not in ("euler", "mixed"):
        kw.update(navier_stokes=1, reynolds=200.0, viscous=hg.BR1 if kind == "br1" else hg.IP, ip_method=hg.SIPG, sigma0_ip=5.0)
    if kind in ("modal", "jumps"):
        kw.update(av_type=hg.AV_LAPLACIAN, av_intensity=1.0)
    g = hg.GpuDGSEM(d, precision=precision, **kw)
    if kind == "modal":
        g.set_sensor(hg.SENSOR_MODAL)
    x = d["x"].reshape(-1, 2)
    return g, cases.kelvin_helmholtz(x[:, 0], x[:, 1], seed=2).ravel()


@pytest.mark.parametrize("precision", [hg.PREC_FP64, hg.PREC_FP32])
@pytest.mark.parametrize("kind", ["euler", "mixed", "br1", "ip", "modal", "jumps"])
def test_waits_that_give_up(kind, precision):
    g, Q = context(kind, precision)
    polls = hg.lib.load().hg_test_copy_polls
    polls.argtypes = [C.c_void_p, C.c_int32]
    g.set_state(Q)
    ref = g.compute_time_derivative(0.0)
    assert polls(g._h, 0) == 0
    with pytest.raises(hg.HorsesGpuError, match="gave up") as ex:
        g.compute_time_derivative(0.0)
    assert ex.value.status == 1 and g.health()[0] == hg.HEALTH_COPY
    g.set_state(Q)
    assert polls(g._h, 0) == 0
    try:
        g.time_step(hg.SCHEME_RK3, 0.0, 1e-5)   # asynchronous
    except hg.HorsesGpuError:
        assert kind in ("ip", "modal")          # the gradient kernel that set_state runs has given up already
    for call in (g.synchronize, g.residuals, lambda: g.time_steps(hg.SCHEME_RK3, 6, 0.0, 1e-5)):
        with pytest.raises(hg.HorsesGpuError, match="gave up") as ex:
            call()
        assert ex.value.status == 1
    assert polls(g._h, -1) == 0
    g.set_state(Q)
    assert g.health() == (0, -1)
    np.testing.assert_array_equal(g.compute_time_derivative(0.0), ref)
    g.time_steps(hg.SCHEME_RK3, 6, 0.0, 1e-5)
    g.synchronize()
    assert g.health() == (0, -1)

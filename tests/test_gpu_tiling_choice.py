"""hg_set_tiling runs the variant it is given on every mesh; a context without one takes variant 1 on a small mesh and
variant 0 on a large one.  Both variants agree (the suite's bounds: relative L2 1e-12 in FP64, 1e-4 in FP32) on 35
elements, which leave the last group of every group size partly empty, for every order, on affine and curved elements."""
import numpy as np
import pytest

import horses2d_b200 as hg
from horses2d_b200 import mesh as hmesh, cases
from cases_util import perturbed, rel_l2

pytestmark = pytest.mark.gpu


def context(N, kind, curved, precision, n=(7, 5)):
    kw = dict(mach=0.3, node_type=hg.NODES_LG, riemann=hg.ROE, precision=precision)
    if kind != "euler":
        kw.update(navier_stokes=1, reynolds=200.0, viscous=hg.BR1 if kind == "br1" else hg.IP, ip_method=hg.SIPG, sigma0_ip=5.0)
    u = np.sqrt(1.4) * 0.3
    stream = np.array([1.0, u, 0.0, 2.5 + 0.5 * u * u])
    if curved:
        d = hmesh.build_descriptor(hmesh.ogrid(*n, 0.5, 8.0, 1.2), N, hg.NODES_LG)
        wall = dict(type=hg.BC_EULERWALL) if kind == "euler" else dict(type=hg.BC_VISCOUSWALL, wall_type=2)
        kw["bcs"] = [wall, dict(type=hg.BC_FARFIELD, state=stream)]
        Q = np.tile(stream, len(d["jac"]))
    else:
        d = hmesh.box_descriptor(*n, 0.0, 1.0, 0.0, 1.0, N, hg.NODES_LG)
        kw["bcs"] = [dict(type=hg.BC_PERIODIC)] * 4
        x = d["x"].reshape(-1, 2)
        Q = cases.kelvin_helmholtz(x[:, 0], x[:, 1], seed=2).ravel()
    return hg.GpuDGSEM(d, **kw), perturbed(Q, 0.01, seed=N)


@pytest.mark.parametrize("precision,tol", [(hg.PREC_FP64, 1e-12), (hg.PREC_FP32, 1e-4)])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("kind,N", [("euler", N) for N in range(1, 13)] + [(k, N) for k in ("br1", "ip") for N in range(1, 11)])
def test_variants_agree_with_partly_empty_groups(kind, N, curved, precision, tol):
    out, sizes = [], []
    for v in range(hg.lib.TILINGS):
        g, Q = context(N, kind, curved, precision)
        g.set_tiling(v)
        t = g.get_tiling()
        assert t["variant"] == v
        sizes.append(t["elements_per_cta"])
        g.set_state(Q)
        qdot, res = g.compute_time_derivative(0.0), g.residuals()
        assert np.allclose(res, np.abs(qdot.reshape(-1, 4)).max(0), rtol=1e-15)
        g.time_steps(hg.SCHEME_RK3, 2, 0.0, 1e-6)
        out.append((qdot, g.state()))
    # (Navier-Stokes order 5 in double has groups of two in both, orders 8 to 10 of one)
    assert sizes[0] > sizes[1] or (kind != "euler" and N >= 5) or (kind == "euler" and N >= 10)
    assert rel_l2(out[0][0], out[1][0]) <= tol and rel_l2(out[0][1], out[1][1]) <= tol


@pytest.mark.parametrize("kind", ["euler", "ip"])
def test_the_choice_without_a_set_variant(kind):
    small, _ = context(4, kind, False, hg.PREC_FP64, n=(8, 8))
    large, _ = context(4, kind, False, hg.PREC_FP64, n=(64, 48))
    per = {}
    for g, v in ((small, 1), (large, 0)):
        t = g.get_tiling()
        assert t["variant"] == v
        per[v] = t["elements_per_cta"]
    for v in (0, 1):
        small.set_tiling(v)
        t = small.get_tiling()
        assert t["variant"] == v and t["elements_per_cta"] == per[v]
    assert per[0] > per[1]


def test_autotune_times_two_kernels_on_a_small_mesh():
    g, Q = context(4, "euler", False, hg.PREC_FP64, n=(8, 8))
    g.set_state(Q)
    r = g.autotune(trials=20)
    per = []
    for v in range(hg.lib.TILINGS):
        g.set_tiling(v)
        per.append(g.get_tiling()["elements_per_cta"])
    assert r["tiling"]["elements_per_cta"] == per[r["chosen"]] and per[0] != per[1]

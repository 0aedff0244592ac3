"""Performance cases of the framework: what a user has it compute, over the range of its workloads.

A case is one of the families below at one size, precision and calling pattern.  ``prepare`` builds what a
user's program holds before its time loop (mesh descriptor, context, initial state), ``run`` makes the calls
of that loop, and ``exact`` evaluates the same scheme in 64 bits with plain torch from the same inputs (mesh
descriptor, initial state, sensor weights).

  euler     periodic isentropic vortex box, Legendre-Gauss or Gauss-Lobatto nodes: the Euler build
  ensemble  many vortex boxes of orders 3-7, packed into one context per order and stepped as a group
  cylinder  Navier-Stokes past a cylinder on a curved O-grid, BR1 (steady loop: a residual check per step)
  shock     Mach-3 standing shock with an entropy wave: HLL, SIPG at Re 0, Laplacian dissipation
  kh        periodic Kelvin-Helmholtz shear layer: Navier-Stokes, SIPG, Laplacian dissipation
  prefine   vortex box with a p-refined centre: two orders, faces between them through mortars
  wall      inviscid flow past a cylinder: IIPG, the reference's interface-jumps dissipation, RK5

The runs in 32 bits return their state in 32 bits: that is what their arithmetic resolves.  Time steps are a
fraction of each case's stability limit, so that a state stays physical over any number of passes.
"""
import functools
import random

import numpy as np
import torch

import horses2d_b200 as hg
from horses2d_b200 import cases as initial
from horses2d_b200 import mesh as hmesh
from horses2d_b200 import sensor as hsensor

GAMMA = 1.4
SCHEMES = {"rk3": hg.SCHEME_RK3, "rk5": hg.SCHEME_RK5}
RIEMANN = {"roe": hg.ROE, "hll": hg.HLL, "lxf": hg.LXF}
ENSEMBLE_ORDERS = (3, 4, 5, 6, 7)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one step of the 16 x 16 vortex per call, as a loop that looks at each step makes it
        dict(name="vortex16_step", family="euler", nx=16, ny=16, N=4, nodes="lgl", riemann="roe",
             precision="fp64", call="step", steps=1),
        # a bare time derivative read back with its residuals (implicit or external time integrators, checks),
        # on an odd mesh at order 6
        dict(name="residual_ragged", family="euler", nx=37, ny=23, N=6, nodes="lg", riemann="hll",
             precision="fp64", call="residual", steps=1),
        # the large inviscid box in the reference's precision
        dict(name="box512", family="euler", nx=512, ny=512, N=4, nodes="lgl", riemann="roe",
             precision="fp64", call="steps", steps=6),
        # a parameter study: 128 vortex boxes of five orders, 32-bit arithmetic
        dict(name="ensemble128", family="ensemble", instances=128, n_lo=8, n_hi=48, precision="fp32", steps=6),
        # external aerodynamics on a curved grid, both precisions
        dict(name="cylinder_fp64", family="cylinder", nr=64, nt=128, N=5, precision="fp64", steps=4),
        dict(name="cylinder_fp32", family="cylinder", nr=64, nt=128, N=5, precision="fp32", steps=4),
        # shock capturing: the reference's precision with the modal sensor, 32 bits with the learned one
        dict(name="shock_fp64", family="shock", nx=512, ny=64, N=3, precision="fp64", sensor="modal", steps=10),
        dict(name="shock_fp32", family="shock", nx=512, ny=64, N=3, precision="fp32", sensor="learned", steps=10),
        # the largest runs: the viscous shear layer at order 7
        dict(name="kh_fp64", family="kh", n=384, N=7, precision="fp64", sensor="modal", steps=4),
        dict(name="kh_fp32", family="kh", n=384, N=7, precision="fp32", sensor="learned", steps=4),
        # p-refinement: orders 5 and 7 and the faces between them, state read back at the end of the run
        dict(name="prefine96", family="prefine", n=96, lo=5, hi=7, precision="fp64", steps=20),
        # the reference's own shock capturing on a curved mesh, five-stage scheme
        dict(name="wall_jumps", family="wall", nr=48, nt=96, N=5, precision="fp64", steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    """One more case of the ranges behind the listed ones."""
    family = rng.choice(["euler", "euler", "ensemble", "cylinder", "shock", "kh", "kh", "prefine", "wall"])
    precision = rng.choice(["fp64", "fp32"])
    sensor = rng.choice(["modal", "learned"])
    if family == "euler":
        N, call = rng.randint(1, 8), rng.choice(["step", "residual", "steps", "steps"])
        most = (300_000 if call == "residual" else 6_000_000) / (N + 1) ** 2
        while True:
            nx, ny = _log(rng, 8, 512), _log(rng, 8, 512)
            if nx * ny <= most:
                break
        return dict(family=family, nx=nx, ny=ny, N=N, nodes=rng.choice(["lg", "lgl"]),
                    riemann=rng.choice(["roe", "hll", "lxf"]), precision=precision, call=call,
                    steps=6 if call == "steps" else 1)
    if family == "ensemble":
        return dict(family=family, instances=_log(rng, 8, 128), n_lo=rng.randint(4, 12), n_hi=rng.randint(16, 48),
                    precision=precision, steps=6)
    if family == "cylinder":
        return dict(family=family, nr=_log(rng, 9, 64), nt=_log(rng, 16, 128), N=rng.randint(2, 6),
                    precision=precision, steps=4)
    if family == "shock":
        return dict(family=family, nx=_log(rng, 64, 512), ny=_log(rng, 4, 80), N=rng.randint(3, 5),
                    precision=precision, sensor=sensor, steps=10)
    if family == "kh":
        return dict(family=family, n=_log(rng, 16, 300), N=rng.randint(3, 7), precision=precision, sensor=sensor,
                    steps=4)
    if family == "prefine":
        lo = rng.randint(3, 6)
        return dict(family=family, n=4 * _log(rng, 5, 28), lo=lo, hi=lo + rng.randint(1, 2), precision="fp64", steps=20)
    return dict(family=family, nr=_log(rng, 9, 56), nt=_log(rng, 16, 112), N=rng.randint(2, 5), precision="fp64", steps=4)


# ------------------------------------------------------------------ inputs
def _boxes(case):
    """(n, N) of an ensemble's boxes: part of the case, not of the seed."""
    r = random.Random(case["instances"] * 1000 + case["n_lo"] * 50 + case["n_hi"])
    return [(r.randint(case["n_lo"], case["n_hi"]), ENSEMBLE_ORDERS[k % 5]) for k in range(case["instances"])]


def _orders(case):
    """Orders of the p-refined box: `hi` in the central half of each direction, `lo` around it."""
    n = case["n"]
    i, j = np.tile(np.arange(n), n), np.repeat(np.arange(n), n)
    inner = (i >= n // 4) & (i < n - n // 4) & (j >= n // 4) & (j < n - n // 4)
    return np.where(inner, case["hi"], case["lo"]).astype(np.int32)


@functools.lru_cache(maxsize=2)
def _mesh(key):
    """Mesh descriptors of a case, one per context (the mesh does not depend on the seed)."""
    case = dict(key)
    f = case["family"]
    if f == "euler":
        return [hmesh.box_descriptor(case["nx"], case["ny"], -5.0, 5.0, -5.0, 5.0, case["N"], _node_type(case))]
    if f == "ensemble":
        out = []
        for N in ENSEMBLE_ORDERS:
            eo = fo = 0
            ds = []
            for n, Nk in _boxes(case):
                if Nk == N:
                    ds.append(hmesh.box_descriptor(n, n, -5.0, 5.0, -5.0, 5.0, N, hg.NODES_LGL, elem_offset=eo,
                                                   edge_offset=fo))
                    eo += len(ds[-1]["N"])
                    fo += len(ds[-1]["edge_marker"])
            out.append(hmesh.concat_descriptors(ds))
        return out
    if f in ("cylinder", "wall"):
        return [hmesh.build_descriptor(hmesh.ogrid(case["nr"], case["nt"], 0.5, 30.0, 1.05), case["N"], hg.NODES_LG)]
    if f == "shock":
        return [hsensor.shock_case(case["nx"], case["ny"], case["N"])[0]]
    if f == "kh":
        return [hmesh.box_descriptor(case["n"], case["n"], 0.0, 1.0, 0.0, 1.0, case["N"], hg.NODES_LG)]
    return [hmesh.box_descriptor(case["n"], case["n"], -5.0, 5.0, -5.0, 5.0, _orders(case), hg.NODES_LG)]


def _node_type(case):
    return hg.NODES_LGL if case.get("nodes") == "lgl" or case["family"] == "ensemble" else hg.NODES_LG


def _freestream(mach):
    u = np.sqrt(GAMMA) * mach
    return np.array([1.0, u, 0.0, 1.0 / (GAMMA - 1.0) + 0.5 * u * u])


def _sensor_weights(seed):
    """A network that answers to the energy in an element's highest modes (features 3, 7, 11, 15: log10 of the
    fraction in the modes of index 3 and above), with seeded noise on every weight; and its feature box."""
    r = np.random.default_rng(seed)
    w1, b1 = r.normal(0.0, 0.01, (32, 16)), r.normal(0.0, 0.01, 32)   # [unit][input]
    w2, b2 = r.normal(0.0, 0.01, (32, 32)), r.normal(0.0, 0.01, 32)
    w3, b3 = r.normal(0.0, 0.01, 32), -1.0
    for k in range(4):
        w1[k, 4 * k + 3], b1[k], w2[k, k], w3[k] = 0.6, 2.4, 1.5, 1.2
    mlp = np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, [b3]]).astype(np.float32)
    return mlp, np.full(16, -12.0, np.float32), np.full(16, 1.0, np.float32)


def _inputs(case, seed):
    """(descriptors, initial states, GpuDGSEM keyword arguments, scheme, dt, sensor weights or None)."""
    f, r = case["family"], np.random.default_rng(seed)
    descs = _mesh(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "call", "precision",
                                                                            "riemann", "sensor"))))
    scheme, mlp = "rk3", None
    if f in ("euler", "ensemble", "prefine"):
        def vortex(d):
            x = d["x"].reshape(-1, 2)
            xc, yc = r.uniform(-1.0, 1.0, 2)
            return initial.isentropic_vortex(x[:, 0], x[:, 1], mach=0.5, beta=r.uniform(3.0, 5.0), xc=xc, yc=yc)
        if f == "ensemble":
            states = []
            for N, d in zip(ENSEMBLE_ORDERS, descs):
                x, o, qs = d["x"].reshape(-1, 2), 0, []
                for n, Nk in _boxes(case):
                    if Nk == N:
                        m = n * n * (N + 1) ** 2
                        qs.append(vortex(dict(x=x[o:o + m])))
                        o += m
                states.append(np.concatenate(qs).ravel())
            h, N = 10.0 / case["n_hi"], 7
        else:
            states = [vortex(descs[0]).ravel()]
            h, N = (10.0 / max(case["nx"], case["ny"]), case["N"]) if f == "euler" else (10.0 / case["n"], case["hi"])
        dt = 0.05 * h / (N + 1) * 0.59 / 2.5
        kw = dict(mach=0.5, node_type=_node_type(case), riemann=RIEMANN[case.get("riemann", "roe")],
                  bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    elif f == "cylinder":
        states = [np.tile(_freestream(0.2), len(descs[0]["jac"])) + 1e-3 * r.standard_normal(4 * len(descs[0]["jac"]))]
        dt = 1.0e-5 * (5.0 / case["N"]) ** 2 * (128.0 / case["nt"]) ** 2
        kw = dict(mach=0.2, reynolds=100.0, prandtl=0.72, navier_stokes=1, viscous=hg.BR1, node_type=hg.NODES_LG,
                  riemann=hg.ROE, bcs=[dict(type=hg.BC_VISCOUSWALL, wall_type=2),
                                       dict(type=hg.BC_FARFIELD, state=_freestream(0.2))])
    elif f == "wall":
        scheme = "rk5"
        states = [np.tile(_freestream(0.4), len(descs[0]["jac"])) + 5e-3 * r.standard_normal(4 * len(descs[0]["jac"]))]
        dt = 1.0e-5 * (5.0 / case["N"]) ** 2 * (96.0 / case["nt"]) ** 2
        kw = dict(mach=0.4, reynolds=0.0, navier_stokes=1, viscous=hg.IP, ip_method=hg.IIPG, sigma0_ip=10.0,
                  node_type=hg.NODES_LG, riemann=hg.HLL, av_type=hg.AV_LAPLACIAN, av_intensity=1.0,
                  bcs=[dict(type=hg.BC_EULERWALL), dict(type=hg.BC_FARFIELD, state=_freestream(0.4))])
    elif f == "shock":
        # a captured shock: the two sides blended over an element's width, so that the sensors have work to do
        x, amp = descs[0]["x"].reshape(-1, 2)[:, 0], r.uniform(0.1, 0.3)
        x_s = hsensor.snap_to_face(5.0 + r.uniform(-0.5, 0.5), case["nx"])
        behind = 0.5 * (1.0 + np.tanh((x - x_s) * case["nx"] / 10.0 / 0.3))[:, None]
        up = hsensor.shock_state(descs[0], 20.0, amp).reshape(-1, 4)
        states = [((1.0 - behind) * up + behind * hsensor.shock_state(descs[0], -20.0).reshape(-1, 4)).ravel()]
        kw = hsensor.shock_case(4, 4, case["N"])[1]
        h = min(10.0 / case["nx"], 1.0 / case["ny"])
        dt = 0.002 * h / (case["N"] + 1) ** 2
    else:
        n, N = case["n"], case["N"]
        xi = descs[0]["x"].reshape(-1, 2)[:N + 1, 0] * n
        states = [initial.kelvin_helmholtz_box(n, N, xi, seed=seed, drho=1.0, delta=max(0.01, 2.0 / n))]
        dt = 0.04 / n ** 2
        kw = dict(mach=0.3, reynolds=1.0e4, navier_stokes=1, viscous=hg.IP, ip_method=hg.SIPG, sigma0_ip=10.0,
                  node_type=hg.NODES_LG, riemann=hg.ROE, av_type=hg.AV_LAPLACIAN, av_intensity=1.0,
                  bcs=[dict(type=hg.BC_PERIODIC)] * 4)
    if case.get("sensor") == "learned":
        mlp = _sensor_weights(seed)
    return descs, states, kw, scheme, dt, mlp


# ------------------------------------------------------------------ the user's program
class _DeviceArray:
    """The resident state of a context as an array that torch can take without a copy; it holds the context,
    so that a tensor taken from it outlives the caller's own reference."""

    def __init__(self, ctx):
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=(ctx.ndof,), typestr="<f8", data=(ctx.device_state_ptr(), False),
                                             version=3)


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


def prepare(case, seed):
    descs, states, kw, scheme, dt, mlp = _inputs(case, seed)
    precision = hg.PREC_FP32 if case["precision"] == "fp32" else hg.PREC_FP64
    ctxs = []
    for d, Q in zip(descs, states):
        g = hg.GpuDGSEM(d, precision=precision, **kw)
        g.set_stream(_stream().cuda_stream)
        if mlp is not None:
            g.set_sensor(hg.SENSOR_LEARNED, mlp=mlp[0], lo=mlp[1], hi=mlp[2])
        elif case.get("sensor") == "modal":
            g.set_sensor(hg.SENSOR_MODAL)
        g.set_state(Q)
        ctxs.append(g)
    s = dict(case=case, ctxs=ctxs, scheme=SCHEMES[scheme], dt=dt)
    if case["family"] == "ensemble":
        s["group"] = hg.GpuGroup(ctxs)
    if case["family"] == "prefine":
        s["host"] = torch.empty(ctxs[0].ndof, dtype=torch.float64).pin_memory().numpy()
    else:
        s["views"] = [torch.as_tensor(_DeviceArray(g), device="cuda") for g in ctxs]
    return s


def _state(s):
    """The resident states as a device-side user (plots, statistics, coupling) takes them."""
    if s["case"]["precision"] == "fp64":
        return s["views"]
    with torch.cuda.stream(_stream()):
        return [v.to(torch.float32) for v in s["views"]]


def run(state):
    case, g = state["case"], state["ctxs"][0]
    f = case["family"]
    if case.get("call") == "residual":
        qdot = g.compute_time_derivative(0.0)
        return [qdot.astype(np.float32) if case["precision"] == "fp32" else qdot]
    if f == "ensemble":
        state["group"].time_steps(state["scheme"], case["steps"], 0.0, state["dt"])
        return _state(state)
    if f == "cylinder":   # a steady run: the residuals decide after each step whether to go on
        for k in range(case["steps"]):
            g.time_step(state["scheme"], k * state["dt"], state["dt"])
            res = g.residuals()
        return _state(state) + [res.astype(np.float32) if case["precision"] == "fp32" else res]
    if case.get("call") == "step":
        g.time_step(state["scheme"], 0.0, state["dt"])
        return _state(state)
    g.time_steps(state["scheme"], case["steps"], 0.0, state["dt"])
    if f == "prefine":
        return [g.state(out=state["host"])]
    return _state(state)


def _nodes(case):
    f = case["family"]
    if f == "euler":
        return case["nx"] * case["ny"] * (case["N"] + 1) ** 2
    if f == "ensemble":
        return sum(n * n * (N + 1) ** 2 for n, N in _boxes(case))
    if f in ("cylinder", "wall"):
        return case["nr"] * case["nt"] * (case["N"] + 1) ** 2
    if f == "shock":
        return case["nx"] * case["ny"] * (case["N"] + 1) ** 2
    if f == "kh":
        return case["n"] ** 2 * (case["N"] + 1) ** 2
    return int(((_orders(case) + 1) ** 2).sum())


def work(case):
    """Bytes: the state in and out once a pass (plus the metrics of curved elements).  Flops: per node and
    stage the two flux contractions, the volume flux, the update and the share of the face fluxes, and for the
    viscous builds the gradient, the viscous fluxes and their face terms."""
    nodes, f = _nodes(case), case["family"]
    P = case.get("N", case.get("hi", 5)) + 1
    stages = case["steps"] * (5 if f == "wall" else 3) if case.get("call") != "residual" else 1
    faces = 4.0 / P   # face nodes per node
    flops = 16.0 * P + 60.0 + 150.0 * faces
    if f in ("cylinder", "kh"):
        flops += 16.0 * P + 100.0 + (200.0 + 32.0 * P) * faces
    curved = f in ("cylinder", "wall")
    return {"bytes": nodes * (64.0 + (40.0 if curved else 0.0)), "flops": nodes * flops * stages}


# ------------------------------------------------------------------ the same scheme in 64 bits, plain torch
def _legendre_nodes(N, lobatto):
    """Nodes and weights on [0, 1] (Gauss, or Gauss-Lobatto: the zeros of the derivative of L_N and the ends)."""
    if not lobatto:
        x, w = np.polynomial.legendre.leggauss(N + 1)
    else:
        c = np.polynomial.legendre.Legendre.basis(N)
        x = np.concatenate([[-1.0], np.sort(c.deriv().roots().real), [1.0]])
        for _ in range(3):   # polish the inner roots
            x[1:-1] -= c.deriv()(x[1:-1]) / c.deriv(2)(x[1:-1])
        w = 2.0 / (N * (N + 1) * c(x) ** 2)
    return 0.5 * (1.0 + x), 0.5 * w


def _interpolation(xi, pts):
    """Lagrange interpolation matrix from nodes xi to points pts."""
    T = np.ones((len(pts), len(xi)))
    for i in range(len(xi)):
        for k in range(len(xi)):
            if k != i:
                T[:, i] *= (pts - xi[k]) / (xi[i] - xi[k])
    return T


class _Order:
    """Nodal operators of one order."""

    def __init__(self, N, lobatto, dev):
        xi, w = _legendre_nodes(N, lobatto)
        P = N + 1
        D = np.zeros((P, P))
        wb = np.array([1.0 / np.prod([xi[j] - xi[k] for k in range(P) if k != j]) for j in range(P)])
        for i in range(P):
            for j in range(P):
                if i != j:
                    D[i, j] = wb[j] / (wb[i] * (xi[i] - xi[j]))
            D[i, i] = -D[i].sum()
        lb = _interpolation(xi, np.array([0.0, 1.0]))
        V = np.stack([np.sqrt(2.0 * k + 1.0) * np.polynomial.legendre.Legendre.basis(k)(2.0 * xi - 1.0)
                      for k in range(P)], 1)
        t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)   # noqa: E731
        self.N, self.P, self.xi, self.w = N, P, xi, w
        self.D, self.hatD = t(D), t((w[:, None] * D).T / w[:, None])
        self.lb, self.lbw, self.dlbw = t(lb), t(lb / w), t(lb @ D / w)
        self.wt, self.Vinv = t(w), t(np.linalg.inv(V))

    def traces(self, Q):
        """[E, eta, xi, ...] -> [E, 4, P, ...]: bottom, right, top, left, each along its own direction."""
        b0, b1 = self.lb[0], self.lb[1]
        return torch.stack([torch.einsum("j,ejik->eik", b0, Q), torch.einsum("i,ejik->ejk", b1, Q),
                            torch.einsum("j,ejik->eik", b1, Q), torch.einsum("i,ejik->ejk", b0, Q)], 1)

    def d_xi(self, M, U):
        return torch.einsum("il,ejlk->ejik", M, U)

    def d_eta(self, M, U):
        return torch.einsum("jl,elik->ejik", M, U)

    def lift(self, F, c):
        """sum over the sides of F (the value at the side node) times the side's column c[0], c[1] across it."""
        return (torch.einsum("eik,j->ejik", F[:, 0], c[0]) + torch.einsum("ejk,i->ejik", F[:, 1], c[1]) +
                torch.einsum("eik,j->ejik", F[:, 2], c[1]) + torch.einsum("ejk,i->ejik", F[:, 3], c[0]))


class _Scheme:
    """The semi-discrete equations of one case."""

    def __init__(self, case, desc, kw, mlp, dev):
        self.case, self.kw, self.mlp, self.dev = case, kw, mlp, dev
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)   # noqa: E731
        lobatto = kw["node_type"] == hg.NODES_LGL
        Ne = np.asarray(desc["N"])
        self.isgm = 1.0 / (np.sqrt(GAMMA) * kw["mach"])
        self.mu = 1.0 / kw["reynolds"] if kw.get("reynolds", 0.0) else 0.0
        self.ns = bool(kw.get("navier_stokes"))
        self.ip = self.ns and kw["viscous"] == hg.IP
        self.eps = {hg.SIPG: -1.0, hg.NIPG: 1.0, hg.IIPG: 0.0}[kw.get("ip_method", hg.SIPG)]
        self.av = kw.get("av_type", hg.AV_NONE) == hg.AV_LAPLACIAN
        el, sd = np.asarray(desc["edge_elem"]).reshape(-1, 2), np.asarray(desc["edge_side"]).reshape(-1, 2) - 1
        mk, inv = np.asarray(desc["edge_marker"]), np.asarray(desc["edge_inverse"])
        n0 = np.concatenate([[0], np.cumsum((Ne + 1) ** 2)])
        PL = Ne[el[:, 0]] + 1
        PR = np.where(mk == 0, Ne[np.maximum(el[:, 1], 0)] + 1, PL)
        PE = np.maximum(PL, PR)
        off = np.concatenate([[0], np.cumsum(PE)])[:-1]
        en, eds = np.asarray(desc["edge_n"]).reshape(-1, 2), np.asarray(desc["edge_dS"])
        periodic = np.array([b["type"] == hg.BC_PERIODIC for b in kw["bcs"]])
        partner = np.asarray(desc["periodic_partner"]) if "periodic_partner" in desc else np.full(len(mk), -1)
        self.parts, local = [], np.zeros(len(Ne), np.int64)
        for N in np.unique(Ne):
            els = np.nonzero(Ne == N)[0]
            local[els] = np.arange(len(els))
            o, P = _Order(int(N), lobatto, dev), int(N) + 1
            nodes = (n0[els][:, None] + np.arange(P * P)[None, :])
            E = len(els)
            p = dict(op=o, E=E, nodes=torch.tensor(nodes, device=dev), N=int(N), els=els)
            p["Ja"] = t(np.asarray(desc["Ja"]).reshape(-1, 4)[nodes].reshape(E, P, P, 4))
            p["J"] = t(np.asarray(desc["jac"])[nodes].reshape(E, P, P, 1))
            p["vol"] = t(np.asarray(desc["volume"])[els])
            self.parts.append(p)
        self.mixed = []
        for p in self.parts:   # side tables: neighbour slot (own where there is none), reversal, LEFT/RIGHT, zone
            P, E, N = p["op"].P, p["E"], p["N"]
            nb, rev = np.zeros((E, 4), np.int64), np.zeros((E, 4), bool)
            right, zone = np.zeros((E, 4), bool), np.full((E, 4), -1)
            geo, invh, per = np.zeros((E, 4, P, 3)), np.zeros((E, 4)), np.zeros((E, 4), bool)
            skip = np.zeros((E, 4), bool)
            ih = np.asarray(desc["edge_invh"]) if "edge_invh" in desc else np.zeros(len(mk))
            rng = np.arange(P)

            def put(f, k, flip):
                e, s = local[el[f, k]], sd[f, k]
                idx = off[f][:, None] + np.where(flip[:, None], P - 1 - rng, rng)
                geo[e, s] = np.concatenate([en[idx], eds[idx][..., None]], -1)
                invh[e, s] = ih[f]
                return e, s
            both = (mk == 0) & (PL == P) & (PR == P)
            f = np.nonzero(both)[0]
            fl = inv[f] != 0
            eL, sL = put(f, 0, np.zeros(len(f), bool))
            eR, sR = put(f, 1, fl)
            nb[eL, sL], rev[eL, sL] = eR * 4 + sR, fl
            nb[eR, sR], rev[eR, sR], right[eR, sR] = eL * 4 + sL, fl, True
            f = np.nonzero((mk != 0) & (PL == P))[0]
            eL, sL = put(f, 0, np.zeros(len(f), bool))
            zone[eL, sL] = mk[f] - 1
            per[eL, sL] = periodic[mk[f] - 1]
            q = np.where(periodic[mk[f] - 1], partner[f], f)
            nb[eL, sL] = local[el[q, 0]] * 4 + sd[q, 0]
            f = np.nonzero((mk == 0) & (PL != PR) & ((PL == P) | (PR == P)))[0]
            k = np.where(PL[f] == P, 0, 1)
            skip[local[el[f, k]], sd[f, k]] = True
            B = lambda a: torch.tensor(a, device=dev)   # noqa: E731
            p.update(nb=B(nb.ravel()), rev=B(rev), right=B(right), zone=zone, per=B(per), geo=t(geo), invh=t(invh),
                     skip=B(skip), bnd=[(z, B(np.argwhere((zone == z) & ~per))) for z in range(len(kw["bcs"]))])
            p["area"] = (p["geo"][..., 2] * p["op"].wt).sum(-1)
            p["interior"] = B((zone < 0) & ~skip)
        for a in range(len(self.parts)):
            for b in range(len(self.parts)):
                pa, pb = self.parts[a], self.parts[b]
                f = np.nonzero((mk == 0) & (PL == pa["op"].P) & (PR == pb["op"].P))[0] if a != b else []
                if len(f):
                    big = max(pa["op"].P, pb["op"].P)
                    idx = off[f][:, None] + np.arange(big)
                    self.mixed.append((a, b, torch.tensor(local[el[f, 0]] * 4 + sd[f, 0], device=dev),
                                       torch.tensor(local[el[f, 1]] * 4 + sd[f, 1], device=dev), t(en[idx]), t(eds[idx])))
        self.mu_held = None

    # ---------------------------------------------------------------- physics
    def pressure(self, q):
        return (GAMMA - 1.0) * (q[..., 3] - 0.5 * (q[..., 1] ** 2 + q[..., 2] ** 2) / q[..., 0])

    def inviscid(self, q):
        r, ru, rv, rE = q.unbind(-1)
        u, v, p = ru / r, rv / r, self.pressure(q)
        return (self.isgm * torch.stack([ru, ru * u + p, ru * v, (rE + p) * u], -1),
                self.isgm * torch.stack([rv, ru * v, rv * v + p, (rE + p) * v], -1))

    def riemann(self, qL, qR, n):
        nx, ny = n[..., 0], n[..., 1]

        def side(q):
            r = q[..., 0]
            u, v = (q[..., 1] * nx + q[..., 2] * ny) / r, (-q[..., 1] * ny + q[..., 2] * nx) / r
            p = self.pressure(q)
            H = (q[..., 3] + p) / r
            return r, u, v, p, H, torch.stack([r, r * u, r * v, q[..., 3]], -1), \
                torch.stack([r * u, r * u * u + p, r * u * v, r * u * H], -1)
        rL, uL, vL, pL, HL, UL, FL = side(qL)
        rR, uR, vR, pR, HR, UR, FR = side(qR)
        sL, sR = torch.sqrt(rL), torch.sqrt(rR)
        u, v, H = ((sL * a + sR * b) / (sL + sR) for a, b in ((uL, uR), (vL, vR), (HL, HR)))
        a = torch.sqrt((GAMMA - 1.0) * (H - 0.5 * (u * u + v * v)))
        kind = self.kw["riemann"]
        if kind == hg.ROE:
            d0, d1, d2, d3 = (UR - UL).unbind(-1)
            a2 = d2 - v * d0
            a1 = (GAMMA - 1.0) * (d0 * (H - u * u) + u * d1 - d3 + a2 * v) / (a * a)
            a0 = (d0 * (u + a) - d1 - a * a1) / (2.0 * a)
            a3 = d0 - (a0 + a1)
            one, zero = torch.ones_like(u), torch.zeros_like(u)
            F = FL
            for lam, al, K in ((u - a, a0, (one, u - a, v, H - u * a)), (u, a1, (one, u, v, 0.5 * (u * u + v * v))),
                               (u, a2, (zero, zero, one, v)), (u + a, a3, (one, u + a, v, H + u * a))):
                F = F + (al * torch.clamp(lam, max=0.0))[..., None] * torch.stack(K, -1)
        else:
            cL, cR = torch.sqrt(GAMMA * pL / rL), torch.sqrt(GAMMA * pR / rR)
            if kind == hg.LXF:
                lam = torch.maximum(uL.abs() + cL, uR.abs() + cR)[..., None]
                F = 0.5 * (FL + FR) - 0.5 * lam * (UR - UL)
            else:
                SL, SR = torch.minimum(uL - cL, u - a)[..., None], torch.maximum(uR + cR, u + a)[..., None]
                mid = (SR * FL - SL * FR + SL * SR * (UR - UL)) / (SR - SL)
                F = torch.where(SL >= 0, FL, torch.where(SR <= 0, FR, mid))
        return self.isgm * torch.stack([F[..., 0], F[..., 1] * nx - F[..., 2] * ny, F[..., 1] * ny + F[..., 2] * nx,
                                        F[..., 3]], -1)

    def viscous(self, q, gx, gy, adiabatic=False):
        """Viscous fluxes per unit viscosity (Stokes hypothesis); adiabatic: without the heat flux."""
        r, u, v = q[..., 0], q[..., 1] / q[..., 0], q[..., 2] / q[..., 0]
        ux, uy = (gx[..., 1] - u * gx[..., 0]) / r, (gy[..., 1] - u * gy[..., 0]) / r
        vx, vy = (gx[..., 2] - v * gx[..., 0]) / r, (gy[..., 2] - v * gy[..., 0]) / r

        def temperature(g):
            return (GAMMA - 1.0) / r * (g[..., 3] - q[..., 3] / r * g[..., 0] + u * (u * g[..., 0] - g[..., 1]) +
                                        v * (v * g[..., 0] - g[..., 2]))
        k = 0.0 if adiabatic else GAMMA / (GAMMA - 1.0) / self.kw.get("prandtl", 0.72)
        txx, tyy, txy = 2.0 * ux - 2.0 / 3.0 * (ux + vy), 2.0 * vy - 2.0 / 3.0 * (ux + vy), uy + vx
        z = torch.zeros_like(u)
        return (torch.stack([z, txx, txy, u * txx + v * txy + k * temperature(gx)], -1),
                torch.stack([z, txy, tyy, u * txy + v * tyy + k * temperature(gy)], -1))

    def boundary(self, z, q, n):
        """(inviscid ghost or None for a prescribed wall flux, viscous state, viscous condition) of zone z."""
        b = self.kw["bcs"][z]
        nx, ny = n[..., 0], n[..., 1]
        r, u, v, p = q[..., 0], q[..., 1] / q[..., 0], q[..., 2] / q[..., 0], self.pressure(q)
        cv = 1.0 / (GAMMA - 1.0)
        if b["type"] == hg.BC_EULERWALL:
            mn, mt = q[..., 1] * nx + q[..., 2] * ny, -q[..., 1] * ny + q[..., 2] * nx
            w = torch.stack([r, q[..., 1] - mn * nx, q[..., 2] - mn * ny, cv * p + 0.5 * mt * mt / r], -1)
            return None, w, "adiabatic"
        if b["type"] == hg.BC_VISCOUSWALL:
            ek = 0.5 * (q[..., 1] ** 2 + q[..., 2] ** 2) / r
            z0 = torch.zeros_like(r)
            return (torch.stack([r, -q[..., 1], -q[..., 2], q[..., 3]], -1),
                    torch.stack([r, z0, z0, q[..., 3] - ek], -1), "adiabatic")
        st = torch.tensor(np.asarray(b["state"], float), dtype=torch.float64, device=q.device).expand_as(q)
        ri, ui, vi, pi = st[..., 0], st[..., 1] / st[..., 0], st[..., 2] / st[..., 0], self.pressure(st)
        un, a = u * nx + v * ny, torch.sqrt(GAMMA * p / r)
        sup = torch.sqrt(u * u + v * v) / a > 1.0
        if b["type"] == hg.BC_DIRICHLET:   # supersonic inflow
            return st, st, "dirichlet"
        if b["type"] == hg.BC_NEWDIRICHLET:   # outflow at the zone's static pressure where subsonic
            ub = torch.stack([r, q[..., 1], q[..., 2], cv * (2.0 * pi - p) + 0.5 * (q[..., 1] * u + q[..., 2] * v)], -1)
            ub = torch.where(sup[..., None], q, ub)
            return ub, ub, "dirichlet"
        pin = 0.5 * (p + pi - r * a * (nx * (u - ui) + ny * (v - vi)))   # far field
        inflow = un < 0.0
        pr = torch.where(inflow, pin, pi)
        rr = torch.where(inflow, ri + (pin - pi) / a ** 2, r + (pi - p) / a ** 2)
        ur = torch.where(inflow, ui + nx * (pin - pi) / (a * r), u - nx * (pi - p) / (a * r))
        vr = torch.where(inflow, vi + ny * (pin - pi) / (a * r), v - ny * (pi - p) / (a * r))
        ub = torch.stack([rr, rr * ur, rr * vr, cv * pr + 0.5 * rr * (ur ** 2 + vr ** 2)], -1)
        ub = torch.where(sup[..., None], torch.where(inflow[..., None], st, q), ub)
        return ub, ub, "neumann"

    # ---------------------------------------------------------------- dissipation
    def ramp(self, s, s0, k):
        return torch.where(s < s0 - k, 0.0, torch.where(s < s0 + k, 0.5 * torch.sin(0.5 * np.pi * (s - s0) / k) + 0.5, 1.0))

    def sensor(self, p, Q):
        """Modal-decay or learned indicator G of each element."""
        o, P = p["op"], p["op"].P
        energy = []
        for v in (Q[..., 0], self.pressure(Q)):
            c = torch.einsum("mi,nj,eji->enm", o.Vinv, o.Vinv, v)
            energy.append(c * c)
        if self.mlp is None:
            s = torch.stack([torch.log10(((c[:, -1].sum(-1) + c[:, :-1, -1].sum(-1)) /
                                          c.sum((1, 2))).clamp(min=1e-30)) for c in energy]).amax(0)
            return self.ramp(s, np.log10(1.0 / P ** 4), 1.0)
        feats = []
        for c in energy:
            tot = c.sum((1, 2))
            for s in (c.sum(1), c.sum(2)):
                s = torch.nn.functional.pad(s, (0, max(0, 4 - P)))
                s = torch.cat([s[:, :3], s[:, 3:].sum(1, keepdim=True)], 1) / tot[:, None]
                feats.append(torch.log10(s.clamp(min=1e-10)))
        x = torch.cat(feats, 1)
        m = torch.tensor(self.mlp[0].astype(np.float64), device=x.device)
        h = torch.tanh(x @ m[:512].view(32, 16).T + m[512:544])
        h = torch.tanh(h @ m[544:1568].view(32, 32).T + m[1568:1600])
        y = torch.sigmoid(h @ m[1600:1632] + m[1632])
        return torch.clamp((y - 0.05) / 0.95, min=0.0)

    def jumps(self, p, tr, nbr, uS):
        """Interface-jumps indicator: per side sum of w (2 (qL - qR) / (qL + qR))^2 dS, for rho and rhoE."""
        other = torch.where(p["interior"][..., None, None] | p["per"][..., None, None], nbr, uS)
        dS = torch.where(p["interior"][..., None], p["geo"][..., 2], p["geo"][:, :, :1, 2])
        g = []
        for k in (0, 3):
            j = 2.0 * (tr[..., k] - other[..., k]) / (tr[..., k] + other[..., k])
            g.append((p["op"].wt * j * j * dS).sum((1, 2)))
        x = torch.maximum(*g) / p["area"].sum(1)
        x = torch.where(x > 1e-8, torch.log10(x.clamp(min=1e-300)), -1e300)
        return self.ramp(x, np.log10(1.0 / p["op"].P ** 4) + 1.0, 5.0)

    # ---------------------------------------------------------------- semi-discrete right-hand side
    def begin_step(self, Qs):
        """Modal and learned indicators hold over a time step."""
        if self.av and self.case["family"] != "wall":
            self.mu_held = [self.viscosity(p, self.sensor(p, Q)) for p, Q in zip(self.parts, Qs)]

    def viscosity(self, p, G):
        return self.kw["av_intensity"] * torch.sqrt(p["vol"]) / p["op"].P * G

    def rhs(self, Qs):
        trs = [p["op"].traces(Q) for p, Q in zip(self.parts, Qs)]
        out = [self.part_rhs(k, p, Q, tr) for k, (p, Q, tr) in enumerate(zip(self.parts, Qs, trs))]
        for a, b, sa, sb, n, dS in self.mixed:   # faces between two orders
            oa, ob = self.parts[a]["op"], self.parts[b]["op"]
            big = oa if oa.P > ob.P else ob
            Ts = [torch.tensor(_interpolation(o.xi, big.xi) if o is not big else np.eye(big.P), dtype=torch.float64,
                               device=self.dev) for o in (oa, ob)]
            q = [torch.einsum("lm,fmk->flk", T, trs[i].reshape(-1, o.P, 4)[s]) for T, i, o, s in
                 zip(Ts, (a, b), (oa, ob), (sa, sb))]
            F = self.riemann(q[0], q[1], n) * dS[..., None]
            for T, i, o, s, sign in zip(Ts, (a, b), (oa, ob), (sa, sb), (1.0, -1.0)):
                out[i][1].view(-1, o.P, 4)[s] = sign * torch.einsum("li,l,flk->fik", T, big.wt, F) / o.wt[:, None]
        return [(vol - p["op"].lift(Fs, p["op"].lbw) - extra) / p["J"] for p, (vol, Fs, extra) in zip(self.parts, out)]

    def part_rhs(self, k, p, Q, tr):
        o, Ja, J, n, dS = p["op"], p["Ja"], p["J"], p["geo"][..., :2], p["geo"][..., 2:]
        J0, J1, J2, J3 = (Ja[..., m:m + 1] for m in range(4))

        def neighbour(T):
            T = T.reshape(-1, o.P, T.shape[-1])[p["nb"]].reshape(T.shape)
            return torch.where(p["rev"][..., None, None], T.flip(2), T)
        nbr = neighbour(tr)
        uB, uS = torch.zeros_like(tr), torch.zeros_like(tr)
        vbc = {}
        wall = torch.zeros(tr.shape[:2], dtype=torch.bool, device=tr.device)
        for z, es in p["bnd"]:
            if len(es):
                e, s = es[:, 0], es[:, 1]
                ghost, uS[e, s], vbc[z] = self.boundary(z, tr[e, s], n[e, s])
                if ghost is None:
                    wall[e, s] = True
                    uB[e, s] = uS[e, s]
                else:
                    uB[e, s] = ghost
        conn = (p["interior"] | p["per"])[..., None, None]
        right = p["right"][..., None, None]
        other = torch.where(conn, nbr, uB)
        qL, qR = torch.where(right, other, tr), torch.where(right, tr, other)
        sign = torch.where(right, -1.0, 1.0)
        Fs = self.riemann(qL, qR, n)
        if wall.any():   # prescribed flux of the state without normal momentum
            fx, fy = self.inviscid(uB)
            Fs = torch.where(wall[..., None, None], fx * n[..., :1] + fy * n[..., 1:], Fs)
        Fs = Fs * sign
        fx, fy = self.inviscid(Q)
        extra = torch.zeros_like(Q)
        if self.ns and (self.mu or self.av):
            need = self.mu != 0.0
            local = torch.cat([(o.d_xi(o.D, Q) * J0 + o.d_eta(o.D, Q) * J1) / J,
                               (o.d_xi(o.D, Q) * J2 + o.d_eta(o.D, Q) * J3) / J], -1)
            grad = local
            if not self.ip:   # BR1: gradient lifted with the face states
                us = torch.where(conn, 0.5 * (tr + nbr), uS) * sign * dS
                fg = torch.cat([us * n[..., :1], us * n[..., 1:]], -1)
                vol = torch.cat([o.d_xi(o.hatD, Q * J0) + o.d_eta(o.hatD, Q * J1),
                                 o.d_xi(o.hatD, Q * J2) + o.d_eta(o.hatD, Q * J3)], -1)
                grad = (o.lift(fg, o.lbw) - vol) / J
            mu_a = None
            if self.av:
                mu_a = self.mu_held[k] if self.mu_held else self.viscosity(p, self.jumps(p, tr, nbr, uS))
                fx, fy = fx - mu_a[:, None, None, None] * local[..., :4], fy - mu_a[:, None, None, None] * local[..., 4:]
                mun = mu_a[:, None].expand(-1, 4).reshape(-1)[p["nb"]].view(-1, 4)
                mu_f = torch.where(p["interior"], 0.5 * (mun + mu_a[:, None]), mu_a[:, None])
                lap = (mu_f * p["area"])[..., None, None]
                Fs = Fs + sign * lap * torch.where(conn, qL - qR, tr - uS)
            if need:
                vx, vy = self.viscous(Q, grad[..., :4], grad[..., 4:])
                fx, fy = fx - self.mu * vx, fy - self.mu * vy
                gt = o.traces(grad)
                gn = neighbour(gt)
                ox, oy = self.viscous(tr, gt[..., :4], gt[..., 4:])
                bx, by = self.viscous(torch.where(conn, nbr, tr), gn[..., :4], gn[..., 4:])
                fv = self.mu * ((0.5 * (ox + bx)) * n[..., :1] + (0.5 * (oy + by)) * n[..., 1:])
                pen = self.kw.get("sigma0_ip", 0.0) * self.mu * o.N ** 2 * p["invh"][..., None, None] if self.ip else 0.0
                fv = fv - pen * (qL - qR)
                G = torch.zeros(tr.shape[:3] + (8,), dtype=tr.dtype, device=tr.device)
                if self.ip and self.eps:
                    jump = qL - qR
                    ax, ay = self.viscous(tr, jump * n[..., :1], jump * n[..., 1:])
                    G = 0.5 * self.eps * self.mu * torch.cat([ax, ay], -1) * dS * sign
                for z, es in p["bnd"]:
                    if len(es):
                        e, s = es[:, 0], es[:, 1]
                        if vbc[z] == "neumann":
                            fv[e, s], G[e, s] = 0.0, 0.0
                            continue
                        wx, wy = self.viscous(tr[e, s], gt[e, s][..., :4], gt[e, s][..., 4:], vbc[z] == "adiabatic")
                        pb = pen[e, s] if self.ip else 0.0
                        fv[e, s] = self.mu * (wx * n[e, s][..., :1] + wy * n[e, s][..., 1:]) - pb * (tr[e, s] - uS[e, s])
                Fs = Fs - sign * fv
                if self.ip and self.eps:
                    Jt, Jat = o.traces(J), o.traces(Ja)
                    c4 = (G[..., :4] * Jat[..., :1] + G[..., 4:] * Jat[..., 2:3]) / Jt
                    c8 = (G[..., :4] * Jat[..., 1:2] + G[..., 4:] * Jat[..., 3:]) / Jt
                    odd = torch.tensor([0, 1, 0, 1], device=tr.device, dtype=torch.bool)[None, :, None, None]
                    along = torch.einsum("kl,eslv->eskv", o.hatD, torch.where(odd, c8, c4))
                    extra = o.lift(along, o.lbw) + o.lift(torch.where(odd, c4, c8), o.dlbw)
        Fs = torch.where(p["skip"][..., None, None], 0.0, Fs * dS)
        vol = o.d_xi(o.hatD, fx * J0 + fy * J2) + o.d_eta(o.hatD, fx * J1 + fy * J3)
        return vol, Fs, extra

    # ---------------------------------------------------------------- state vectors
    def split(self, Q):
        q = torch.tensor(Q, dtype=torch.float64, device=self.dev).view(-1, 4)
        return [q[p["nodes"]].view(p["E"], p["op"].P, p["op"].P, 4) for p in self.parts]

    def join(self, Qs):
        out = torch.empty(sum(Q.numel() for Q in Qs) // 4, 4, dtype=torch.float64, device=self.dev)
        for p, Q in zip(self.parts, Qs):
            out[p["nodes"].reshape(-1)] = Q.reshape(-1, 4)
        return out.reshape(-1)


def _advance(scheme, S, Qs, steps, dt):
    """Low-storage Runge-Kutta steps; returns the states and the last stage's time derivative."""
    a, b, c = {"rk3": ((0.0, -5.0 / 9.0, -153.0 / 128.0), 1.0, tuple(dt * g for g in (1.0 / 3.0, 15.0 / 16.0, 8.0 / 15.0))),
               "rk5": ((0.0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257), dt,
                       (0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488, 0.1530572479681))}[scheme]
    G = [torch.zeros_like(Q) for Q in Qs]
    R = None
    for _ in range(steps):
        S.begin_step(Qs)
        for m in range(len(a)):
            R = S.rhs(Qs)
            G = [a[m] * g + b * r for g, r in zip(G, R)]
            Qs = [Q + c[m] * g for Q, g in zip(Qs, G)]
    return Qs, R


def exact(case, seed):
    descs, states, kw, scheme, dt, mlp = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out, res = [], []
    for d, Q in zip(descs, states):
        S = _Scheme(case, d, kw, mlp, dev)
        Qs = S.split(Q)
        if case.get("call") == "residual":
            return [S.join(S.rhs(Qs)).cpu()]
        Qs, R = _advance(scheme, S, Qs, case["steps"], dt)
        out.append(S.join(Qs).cpu())
        res.append(torch.stack([r.abs().amax((0, 1, 2)) for r in R]).amax(0).cpu())
    return out + (res if case["family"] == "cylinder" else [])

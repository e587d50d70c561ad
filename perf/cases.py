"""The work that the framework is timed on, as a user's program asks for it.

Each listed case is one call (or one short loop) through the public entry
points: a bound right-hand side, an LSRK4 step, the graph-captured time loop,
the gradients, the batched ensemble and the over-integrated advection, over
the orders, sizes, models and precisions that the tests, the benchmark and
the workloads of this repository use.  ``draw`` gives more of the same.

The ``exact`` half is a plain torch evaluation of the same discontinuous
Galerkin operators in 64 bits: element matrices by numerical quadrature,
face nodes matched by their vertices, gradients by torch.autograd.
"""

import itertools
import math

import numpy as np
import torch

import hedge_b200 as hb
from hedge_b200 import adjoint, ensemble

# ---------------------------------------------------------------------------
# cases


def listed():
    return [
        # the 2D reference configuration: advection on 3200 periodic
        # triangles, one step; five launches of a few microseconds
        dict(name="advection2d_step", kind="step", model="advection", dim=2, n=40, m=40, order=4,
             precision="fp64", flux="upwind", bc="periodic"),
        # a small mesh in a time loop with an energy log: a recorded step
        # replayed ten times, then the norm of the state
        dict(name="wave2d_loop", kind="loop", model="wave", dim=2, n=18, m=19, order=3,
             precision="fp64", flux="upwind", bc="open", steps=10),
        # one right-hand side of the 2D TM system (an integrator of the
        # user's own), an absorbing side
        dict(name="tm2d_rhs", kind="rhs", model="tm", dim=2, n=97, m=101, order=5,
             precision="fp64", flux="upwind", bc="open"),
        # the headline workload: 3D Maxwell cavity, split FP16 products
        dict(name="maxwell3d_n4_fp16x3_step", kind="step", model="maxwell", dim=3, n=20, m=20,
             order=4, precision="fp16x3", flux="upwind", bc="wall"),
        # the same mesh in the default precision
        dict(name="maxwell3d_n4_fp64_step", kind="step", model="maxwell", dim=3, n=20, m=20,
             order=4, precision="fp64", flux="upwind", bc="wall"),
        # FP32 on a ragged mid-size mesh
        dict(name="maxwell3d_n3_fp32_step", kind="step", model="maxwell", dim=3, n=11, m=13,
             order=3, precision="fp32", flux="lf", bc="open"),
        # high order, split products: the large acoustic pulse
        dict(name="wave3d_n7_fp16x3_step", kind="step", model="wave", dim=3, n=20, m=20, order=7,
             precision="fp16x3", flux="upwind", bc="wall"),
        # low order with spatially variable material
        dict(name="material3d_n2_step", kind="step", model="material", dim=3, n=12, m=15, order=2,
             precision="fp64", flux="upwind", bc="open"),
        # reverse mode through one right-hand side: state and wave speed
        dict(name="varwave2d_grad", kind="grad", model="varwave", dim=2, n=60, m=60, order=5,
             precision="fp64", flux="upwind", bc="wall"),
        # inversion: a short checkpointed time loop with receivers, forward
        # and backward
        dict(name="varwave2d_traces", kind="traces", model="varwave", dim=2, n=32, m=33, order=4,
             precision="fp64", flux="upwind", bc="wall", steps=8, every=4),
        # a parameter study: many members of mixed order and size at once
        dict(name="ensemble2d_step", kind="ensemble", model="mixed", dim=2, members=20, kmin=500,
             kmax=20000, order=6, precision="fp32", flux="upwind", bc="mixed"),
        # over-integrated advection by a rotating velocity
        dict(name="varadv2d_n5_step", kind="step", model="varadv", dim=2, n=200, m=200, order=5,
             precision="fp64", flux="upwind", bc="given"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, dim, order, fields, kmin, most):
    """Cell counts (n, m): K log-uniform from kmin up to `most` unknowns."""
    per = math.comb(order + dim, dim) * fields
    k = math.exp(rng.uniform(math.log(kmin), math.log(max(kmin + 1, min(most / per, 48000)))))
    n = max(4 if dim == 2 else 2, int(round((k / 2) ** 0.5 if dim == 2 else (k / 6) ** (1 / 3))))
    return n, max(4 if dim == 2 else 2, n + rng.randint(-1, 2))


def draw(rng):
    what = rng.choice(["advection", "wave2d", "wave3d", "maxwell", "maxwell", "tmte", "material",
                       "loop", "grad", "traces", "ensemble", "varadv"])
    flux = rng.choice(["upwind", "upwind", "central"])
    bc = rng.choice(["wall", "open"])
    call = rng.choice(["step", "step", "rhs"])
    if what == "advection":
        dim = rng.choice([2, 3])
        order = rng.randint(2, 6)
        n, m = _cells(rng, dim, order, 1, 400, 3e6)
        return dict(kind=call, model="advection", dim=dim, n=n, m=m, order=order,
                    precision=rng.choice(["fp64", "fp64", "fp32"]),
                    flux=rng.choice(["upwind", "lf", "central"]),
                    bc=rng.choice(["periodic", "given"]) if dim == 2 else "given")
    if what == "wave2d":
        order = rng.randint(2, 7)
        n, m = _cells(rng, 2, order, 3, 400, 4e6)
        return dict(kind=call, model="wave", dim=2, n=n, m=m, order=order,
                    precision=rng.choice(["fp64", "fp64", "fp32"]), flux=flux, bc=bc)
    if what == "wave3d":
        order = rng.randint(2, 7)
        n, m = _cells(rng, 3, order, 4, 400, 6e6)
        return dict(kind="step", model="wave", dim=3, n=n, m=m, order=order,
                    precision=rng.choice(["fp64", "fp16x3", "fp32"]), flux=flux, bc=bc)
    if what == "maxwell":
        order = rng.randint(2, 5)
        n, m = _cells(rng, 3, order, 6, 400, 6e6)
        return dict(kind=call, model="maxwell", dim=3, n=n, m=m, order=order,
                    precision=rng.choice(["fp64", "fp64", "fp16x3", "fp32"]),
                    flux=rng.choice(["upwind", "lf", "central"]), bc=bc)
    if what == "tmte":
        order = rng.randint(2, 7)
        n, m = _cells(rng, 2, order, 3, 400, 4e6)
        return dict(kind=call, model=rng.choice(["tm", "te"]), dim=2, n=n, m=m, order=order,
                    precision=rng.choice(["fp64", "fp64", "fp32"]),
                    flux=rng.choice(["upwind", "lf", "central"]), bc=bc)
    if what == "material":
        order = rng.randint(2, 4)
        n, m = _cells(rng, 3, order, 6, 400, 3e6)
        return dict(kind=call, model="material", dim=3, n=n, m=m, order=order, precision="fp64",
                    flux=rng.choice(["upwind", "lf"]), bc=bc)
    if what == "loop":
        dim = rng.choice([2, 3])
        order = rng.randint(2, 4)
        n, m = _cells(rng, dim, order, dim + 1, 128, 2e5)
        return dict(kind="loop", model="wave", dim=dim, n=n, m=m, order=order, precision="fp64",
                    flux=flux, bc=bc, steps=rng.randint(4, 16))
    if what == "grad":
        model, dim = rng.choice([("varwave", 2), ("varwave", 3), ("maxwell", 3), ("wave", 2)])
        order = rng.randint(2, 6 if dim == 2 else 4)
        n, m = _cells(rng, dim, order, 6 if model == "maxwell" else dim + 1, 400, 1e6)
        return dict(kind="grad", model=model, dim=dim, n=n, m=m, order=order, precision="fp64",
                    flux="upwind", bc=bc)
    if what == "traces":
        order = rng.randint(2, 6)
        n, m = _cells(rng, 2, order, 3, 400, 2e5)
        return dict(kind="traces", model="varwave", dim=2, n=n, m=m, order=order,
                    precision="fp64", flux="upwind", bc="wall", steps=rng.randint(3, 10),
                    every=rng.randint(2, 5))
    if what == "ensemble":
        return dict(kind="ensemble", model="mixed", dim=2, members=rng.randint(3, 20), kmin=500,
                    kmax=_log_int(rng, 2000, 20000), order=rng.randint(4, 6), precision="fp32",
                    flux="upwind", bc="mixed")
    order = rng.randint(2, 5)
    n, m = _cells(rng, 2, order, 1, 400, 1e6)
    return dict(kind="step", model="varadv", dim=2, n=n, m=m, order=order,
                precision=rng.choice(["fp64", "fp64", "fp32"]),
                flux=rng.choice(["upwind", "lf", "central"]), bc="given")


# ---------------------------------------------------------------------------
# inputs, from the seed alone


def _fields(case):
    return {"advection": 1, "varadv": 1, "wave": case["dim"] + 1, "varwave": case["dim"] + 1,
            "maxwell": 6, "material": 6, "tm": 3, "te": 3}[case["model"]]


def _mesh(case, seed):
    """Jittered box mesh on [-1, 1]^d; its boundary faces carry "wall",
    "open" (the side x = 1), "inflow" and "outflow"."""
    n, m, bc = case["n"], case["m"], case["bc"]

    def tagger(fvi, el, fn, points):
        c = points[list(fvi)].mean(axis=0)
        return ["inflow" if np.any(np.abs(c + 1) < 1e-9) else "outflow",
                "open" if bc == "open" and abs(c[0] - 1) < 1e-9 else "wall"]

    jitter = 0.1 * 2.0 / max(n, m)
    if case["dim"] == 2:
        return hb.make_regular_rect_mesh((-1, -1), (1, 1), (n + 1, m + 1), jitter=jitter,
                                         seed=seed, boundary_tagger=tagger,
                                         periodicity=(bc == "periodic",) * 2)
    return hb.make_box_tet_mesh(n=(n, n, m), jitter=jitter, seed=seed, boundary_tagger=tagger)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _smooth(x, fields, rng):
    """[fields, len(x)] smooth modes plus 1e-3 noise (x: [N, d] on the device)."""
    gen = torch.Generator(device=x.device).manual_seed(int(rng.integers(1 << 31)))
    out = torch.empty((fields, len(x)), dtype=torch.float64, device=x.device)
    for f in range(fields):
        k = torch.as_tensor(math.pi * rng.integers(1, 4, (2, x.shape[1])), device=x.device,
                            dtype=torch.float64)
        ph = rng.uniform(0, 2 * math.pi, 2)
        out[f] = sum(torch.cos(x @ k[i] + float(ph[i])) for i in range(2)) * 0.5
    noise = torch.rand(out.shape, generator=gen, dtype=torch.float64, device=x.device)
    return out + 1e-3 * (2 * noise - 1)


def _velocity(x):
    return np.stack([-x[:, 1], x[:, 0]])


def _inflow(x):
    return np.cos(2 * x.sum(axis=1))


def _amplitude(t):
    return math.cos(8 * t)


def _advection_v(dim):
    return np.array([1.0, 0.5, 0.25][:dim])


def _inputs(case, seed):
    """Mesh, node coordinates and volume vectors of a case."""
    rng = np.random.default_rng(seed)
    mesh = _mesh(case, int(rng.integers(1 << 30)))
    x = _nodes(mesh, case["order"])
    w = _smooth(x, _fields(case), rng)
    inp = dict(mesh=mesh, x=x, w=w)
    if case["precision"] == "fp32":
        inp["w"] = w.float()
    if case["model"] == "varwave":
        inp["c"] = 1.0 + 0.2 * _smooth(x, 1, rng)[0]
    if case["model"] == "material":
        s = _smooth(x, 2, rng)
        inp["eps"], inp["mu"] = 1.5 + 0.4 * s[0], 1.2 + 0.3 * s[1]
    if case["kind"] == "grad":
        inp["lam"] = _smooth(x, _fields(case), rng)
    if case["kind"] == "traces":
        inp["points"] = rng.uniform(-0.8, 0.8, (16, 2))
        inp["source"] = torch.exp(-(x ** 2).sum(1) / 0.1 ** 2)
    return inp


def _operator(case, inp):
    dim, model, flux = case["dim"], case["model"], case["flux"]
    if model == "advection":
        return hb.StrongAdvectionOperator(_advection_v(dim), flux_type=flux,
                                          inflow_u=hb.TimeConstantGivenFunction(_inflow))
    if model == "varadv":
        return hb.VariableCoefficientAdvectionOperator(
            dim, hb.TimeConstantGivenFunction(_velocity),
            bc_u_f=hb.TimeConstantGivenFunction(_inflow), flux_type=flux)
    if model == "wave":
        return hb.StrongWaveOperator(1.0, dim, flux_type=flux, dirichlet_tag="wall",
                                     radiation_tag="open")
    if model == "varwave":
        return hb.VariableVelocityStrongWaveOperator(inp["c"], dim, flux_type=flux,
                                                     dirichlet_tag="wall", radiation_tag="open")
    cls = {"tm": hb.TMMaxwellOperator, "te": hb.TEMaxwellOperator}.get(model, hb.MaxwellOperator)
    eps, mu = (inp["eps"], inp["mu"]) if model == "material" else (1.0, 1.0)
    return cls(eps, mu, flux_type={"upwind": 1, "central": 0}.get(flux, flux), pec_tag="wall",
               absorb_tag="open")


def _members(case, seed):
    """Specifications of the ensemble's members and their initial states."""
    rng = np.random.default_rng(seed)
    spread = np.linspace(math.log(case["kmin"]), math.log(case["kmax"]), case["members"])
    out = []
    for k in range(case["members"]):
        n = max(4, int(round(math.sqrt(math.exp(spread[k]) / 2))))
        model = ("advection", "wave")[k % 2]
        c = dict(kind="step", model=model, dim=2, n=n, m=n + 1, order=3 + k % (case["order"] - 2),
                 precision="fp32", flux="upwind", bc="periodic" if k % 2 == 0 else "wall")
        out.append((c, int(rng.integers(1 << 30))))
    return out


def _time_step(case):
    """About 0.4 of the CFL estimate for unit speed, from the sizes alone."""
    return 0.5 * (2.0 / max(case["n"], case["m"])) / (case["order"] + 1) ** 2


def prepare(case, seed):
    if case["kind"] == "ensemble":
        members = []
        for c, s in _members(case, seed):
            inp = _inputs(c, s)
            discr = hb.Discretization(inp["mesh"], order=c["order"])
            members.append(ensemble.Member(discr, _operator(c, inp), inp["w"].cpu().numpy(),
                                           dt=_time_step(c)))
        ens = ensemble.Ensemble(members)
        ens.capture()
        return dict(case=case, ens=ens)
    inp = _inputs(case, seed)
    quad = {"quad": 3 * case["order"]} if case["model"] == "varadv" else None
    discr = hb.Discretization(inp["mesh"], order=case["order"], precision=case["precision"],
                              quad_min_degrees=quad)
    rhs = _operator(case, inp).bind(discr)
    st = dict(case=case, discr=discr, rhs=rhs, w=inp["w"], dt=_time_step(case))
    if case["kind"] == "step":
        st["stepper"] = hb.LSRK4TimeStepper()
    elif case["kind"] == "loop":
        st["graph"] = hb.GraphedLSRK4(rhs, inp["w"], st["dt"])
    elif case["kind"] == "grad":
        st["w"] = inp["w"].requires_grad_(True)
        st["c"] = inp["c"].requires_grad_(True) if "c" in inp else None
        st["lam"] = inp["lam"]
    elif case["kind"] == "traces":
        st["w"] = inp["w"].requires_grad_(True)
        st["c"] = inp["c"].requires_grad_(True)
        st["receivers"] = adjoint.Receivers(discr, inp["points"])
        st["source"] = (inp["source"], _amplitude)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rhs":
        return state["rhs"](0.0, state["w"])
    if kind == "step":
        return state["stepper"](state["w"], 0.0, state["dt"], state["rhs"])
    if kind == "loop":
        g = state["graph"]
        for _ in range(case["steps"]):
            y = g.step()
        return y, state["discr"].norm(y)
    if kind == "grad":
        w, c = state["w"], state["c"]
        out = adjoint.RHSFunction.apply(w, c, state["rhs"].compiled)
        grads = torch.autograd.grad(out, [w] if c is None else [w, c], state["lam"])
        return [out.detach(), *grads]
    if kind == "traces":
        w, c = state["w"], state["c"]
        traces = adjoint.ReceiverTraces.apply(w, c, state["rhs"].compiled, state["receivers"],
                                              state["dt"], case["steps"], state["source"],
                                              case["every"])
        grads = torch.autograd.grad(adjoint.trace_loss(traces), [w, c])
        return [traces.detach(), *grads]
    ens = state["ens"]
    ens.step(1)
    return [ens.state(k) for k in range(case["members"])]


def _counts(case):
    dim, n = case["dim"], case["order"]
    k = 2 * case["n"] * case["m"] if dim == 2 else 6 * case["n"] ** 2 * case["m"]
    return k, math.comb(n + dim, dim), (dim + 1) * math.comb(n + dim - 1, dim - 1)


def work(case):
    """Per stage: the state and the residual read and written once (FP32
    states of the ensemble with an FP64 residual), the geometry and the face
    table read; the arithmetic of the element matrices."""
    if case["kind"] == "ensemble":
        tot = dict(bytes=0.0, flops=0.0)
        for c, _ in _members(case, 0):
            k, np_, nfpt = _counts(c)
            f = _fields(c)
            tot["bytes"] += 5 * k * (np_ * f * 24 + 4 * 13 + 8 * 3)
            tot["flops"] += 5 * k * f * (4 * np_ * np_ + 2 * np_ * nfpt)
        return tot
    dim, f = case["dim"], _fields(case)
    k, np_, nfpt = _counts(case)
    size = 4 if case["precision"] == "fp32" else 8
    geo = size * (dim * dim + (dim + 1) ** 2) + 8 * (dim + 1)
    extra = {"varwave": 1, "material": 2, "varadv": dim}.get(case["model"], 0) * 8 * np_
    rhs_flops = k * f * (2 * dim * np_ * np_ + 2 * np_ * nfpt)
    if case["model"] == "varadv":
        # exact volume rule and face rule of the integrand's degree
        nq, nqf = ((3 * case["order"] + 1) // 2) ** 2, (3 * case["order"]) // 2 + 1
        nfp = case["order"] + 1
        rhs_flops = 2 * k * ((1 + dim) * nq * np_ + dim * nq * np_
                             + 3 * (2 * (1 + dim) * nqf * nfp + nqf * np_))
    stage = k * (np_ * f * 4 * size + geo + extra)
    once = k * (np_ * f * 2 * size + geo + extra)
    kind = case["kind"]
    if kind == "rhs":
        return dict(bytes=float(once), flops=float(rhs_flops))
    if kind == "step":
        return dict(bytes=5.0 * stage, flops=5.0 * rhs_flops)
    if kind == "loop":
        return dict(bytes=5.0 * case["steps"] * stage, flops=5.0 * case["steps"] * rhs_flops)
    if kind == "grad":
        c = 8 * np_ if case["model"] == "varwave" else 0
        return dict(bytes=float(2 * once + k * (np_ * f * 8 + c)),
                    flops=float(rhs_flops * (3 if c else 2)))
    # traces: forward, recomputed forward, adjoint stages
    s = 5.0 * case["steps"]
    return dict(bytes=s * (2 * stage + once + k * np_ * (f + 1) * 8), flops=s * 5 * rhs_flops)


# ---------------------------------------------------------------------------
# the same operators in plain torch, 64 bits

_ALPHA = {2: [0.0, 0.0, 1.4152, 0.1001, 0.2751, 0.98, 1.0999],
          3: [0.0, 0.0, 0.0, 0.1002, 1.1332, 1.5608, 1.3413]}
_FACES = {2: [(0, 1), (1, 2), (0, 2)], 3: [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)]}
_LSRK_A = [0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238,
           -3550918686646 / 2091501179385, -1275806237668 / 842570457699]
_LSRK_B = [1432997174477 / 9575080441755, 5161836677717 / 13612068292357,
           1720146321549 / 2090206949498, 3134564353537 / 4481467310338,
           2277821191437 / 14882151754819]
_LSRK_C = [0.0, 1432997174477 / 9575080441755, 2526269341429 / 6820363962896,
           2006345519317 / 3224310063776, 2802321613138 / 2924317926251]


def _tuples(order, dim):
    """Node numbering: index tuples of sum <= order, the first fastest."""
    t = [x[::-1] for x in itertools.product(range(order + 1), repeat=dim)]
    return np.array([x for x in t if sum(x) <= order])


def _gauss_simplex(dim, n):
    """Points and weights on the biunit simplex, collapsed Gauss-Legendre."""
    a, wa = np.polynomial.legendre.leggauss(n)
    if dim == 1:
        return a[:, None], wa
    if dim == 2:
        A, B = np.meshgrid(a, a, indexing="ij")
        W = np.outer(wa, wa * (1 - a) / 2)
        return np.stack([((1 + A) * (1 - B) / 2 - 1).ravel(), B.ravel()], 1), W.ravel()
    A, B, C = np.meshgrid(a, a, a, indexing="ij")
    W = np.einsum("i,j,k->ijk", wa, wa * (1 - a) / 2, wa * ((1 - a) / 2) ** 2)
    x = np.stack([((1 + A) * (1 - B) * (1 - C) / 4 - 1).ravel(),
                  ((1 + B) * (1 - C) / 2 - 1).ravel(), C.ravel()], 1)
    return x, W.ravel()


def _warp_blend(order, dim):
    """Warburton's warp-and-blend nodes on the biunit simplex."""
    tup = _tuples(order, dim) / order
    lam = np.concatenate([1 - tup.sum(1, keepdims=True), tup], 1)
    eq = np.linspace(-1, 1, order + 1)
    inner = np.polynomial.legendre.Legendre.basis(order).deriv().roots() if order > 1 else []
    gap = np.concatenate([[-1.0], np.sort(inner), [1.0]]) - eq

    def warp(x):
        y = np.zeros_like(x)
        for i in range(order + 1):
            y = y + gap[i] * np.prod([(x - eq[j]) / (eq[i] - eq[j])
                                      for j in range(order + 1) if j != i], axis=0)
        inside = np.abs(x) < 1 - 1e-10
        return np.where(inside, y / np.where(inside, 1 - x * x, 1.0), 0.0)

    def tri_shift(b, alpha):
        v = np.array([[-1, -1 / 3 ** 0.5], [1, -1 / 3 ** 0.5], [0, 2 / 3 ** 0.5]])
        s = 0.0
        for (i, j), o in (((0, 1), 2), ((1, 2), 0), ((0, 2), 1)):
            e = (v[j] - v[i]) / np.linalg.norm(v[j] - v[i])
            amount = 4 * b[:, i] * b[:, j] * warp(b[:, j] - b[:, i]) * (1 + (alpha * b[:, o]) ** 2)
            s = s + amount[:, None] * e
        return s

    alpha = _ALPHA[dim][order - 1]
    if dim == 2:
        v = np.array([[-1, -1 / 3 ** 0.5], [1, -1 / 3 ** 0.5], [0, 2 / 3 ** 0.5]])
        x = lam @ v + tri_shift(lam, alpha)
    else:
        r3, r6 = 3 ** 0.5, 6 ** 0.5
        v = np.array([[-1, -1 / r3, -1 / r6], [1, -1 / r3, -1 / r6], [0, 2 / r3, -1 / r6],
                      [0, 0, 3 / r6]])
        x = lam @ v
        for f in _FACES[3]:
            o = 6 - sum(f)
            d1 = v[f[1]] - v[f[0]]
            d2 = v[f[2]] - (v[f[0]] + v[f[1]]) / 2
            den = np.stack([lam[:, i] + 0.5 * lam[:, o] for i in f])
            ok = np.all(np.abs(den) > 1e-12, axis=0)
            blend = np.where(ok, lam[:, f[0]] * lam[:, f[1]] * lam[:, f[2]]
                             * (1 + alpha * lam[:, o]) ** 2
                             / np.where(ok, np.prod(den, axis=0), 1.0), 0.5)
            s = tri_shift(lam[:, list(f)], alpha) * blend[:, None]
            x = x + s[:, :1] * d1 / np.linalg.norm(d1) + s[:, 1:] * d2 / np.linalg.norm(d2)
    # equilateral -> biunit: affine, by the vertices
    unit = np.concatenate([-np.ones((1, dim)), 2 * np.eye(dim) - 1])
    aff = np.linalg.solve(np.concatenate([v, np.ones((dim + 1, 1))], 1), unit)
    return x @ aff[:dim] + aff[dim]


class _Element:
    """Nodal basis of an order on the simplex, its matrices by quadrature."""

    cache = {}

    def __new__(cls, order, dim):
        if (order, dim) not in cls.cache:
            self = cls.cache[order, dim] = super().__new__(cls)
            self.build(order, dim)
        return cls.cache[order, dim]

    def build(self, order, dim):
        self.order, self.dim = order, dim
        self.tup = _tuples(order, dim)
        self.nodes = _warp_blend(order, dim)
        q, wq = _gauss_simplex(dim, order + 2)
        r = np.eye(len(self.tup))
        for _ in range(2):   # orthonormalise twice
            r = r @ np.linalg.inv(np.linalg.qr(np.sqrt(wq)[:, None] * (self.modes(q) @ r))[1])
        self.to_modes = r
        self.vinv = np.linalg.inv(self.modes(self.nodes) @ r)
        self.minv = np.linalg.inv(self.vinv.T @ self.vinv)
        self.d = np.stack([self.modes(self.nodes, x) @ r @ self.vinv for x in range(dim)])
        full = np.concatenate([order - self.tup.sum(1, keepdims=True), self.tup], 1)
        vert = np.concatenate([-np.ones((1, dim)), 2 * np.eye(dim) - 1])
        self.fnodes, lift = [], []
        p, wp = _gauss_simplex(dim - 1, order + 2)
        bary = np.concatenate([1 - (p + 1).sum(1, keepdims=True) / 2, (p + 1) / 2], 1)
        for f in _FACES[dim]:
            o = (set(range(dim + 1)) - set(f)).pop()
            idx = np.nonzero(full[:, o] == 0)[0]
            phi = self.phi(bary @ vert[list(f)])
            lift.append(self.minv @ (phi.T * wp) @ phi[:, idx])
            self.fnodes.append(idx)
        self.fnodes = np.array(self.fnodes)
        self.lift = np.concatenate(lift, 1)
        # canonical order of each face's nodes, by how its vertices rank
        self.canon = {}
        for f, verts in enumerate(_FACES[dim]):
            for perm in itertools.permutations(range(dim)):
                key = full[self.fnodes[f]][:, [verts[i] for i in perm]]
                self.canon[f, perm] = np.lexsort(key.T)

    def modes(self, x, diff=None):
        """Products of Legendre polynomials at x (or their derivative)."""
        out = 1.0
        for a in range(self.dim):
            cols = []
            for k in range(self.order + 1):
                p = np.polynomial.legendre.Legendre.basis(k)
                cols.append((p.deriv() if a == diff else p)(x[:, a]))
            out = out * np.stack(cols, 1)[:, self.tup[:, a]]
        return out

    def phi(self, x, diff=None):
        """[points, Np]: the nodal basis (or a derivative) at points."""
        return self.modes(x, diff) @ self.to_modes @ self.vinv


def _maps(mesh):
    v = mesh.points[mesh.elements]
    d = v.shape[2]
    a = 0.5 * (v[:, 1:] - v[:, :1]).transpose(0, 2, 1)
    return v, a, 0.5 * v[:, 1:].sum(1) - 0.5 * (d - 2) * v[:, 0]


def _nodes(mesh, order):
    _, a, b = _maps(mesh)
    dev = _dev()
    r = torch.as_tensor(_Element(order, mesh.points.shape[1]).nodes, device=dev)
    a, b = torch.as_tensor(a, device=dev), torch.as_tensor(b, device=dev)
    return (torch.einsum("kxr,nr->knx", a, r) + b[:, None]).reshape(-1, a.shape[1])


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


class _Plain:
    """The right-hand side of a case's model in plain torch."""

    def __init__(self, case, inp):
        self.case, dim, order = case, case["dim"], case["order"]
        mesh, dev = inp["mesh"], _dev()
        E = self.E = _Element(order, dim)
        v, a, _ = _maps(mesh)
        self.K, self.Np, self.nf = len(v), len(E.nodes), dim + 1

        def t(x):
            return torch.as_tensor(np.ascontiguousarray(x), device=dev)

        self.t = t
        self.inv, jac = t(np.linalg.inv(a)), np.abs(np.linalg.det(a))
        fv = v[:, _FACES[dim]]                                     # [K, nf, dim, d]
        e = fv[:, :, 1:] - fv[:, :, :1]
        if dim == 2:
            n = np.stack([e[..., 0, 1], -e[..., 0, 0]], -1)
            area = np.linalg.norm(n, axis=-1)
        else:
            n = np.cross(e[..., 0, :], e[..., 1, :])
            area = 0.5 * np.linalg.norm(n, axis=-1)
        opp = v[:, [(set(range(dim + 1)) - set(f)).pop() for f in _FACES[dim]]]
        n = n * np.sign(((fv[:, :, 0] - opp) * n).sum(-1))[..., None]
        n = n / np.linalg.norm(n, axis=-1)[..., None]
        self.n = [t(n[..., x])[..., None] for x in range(dim)]
        self.fscale = t(area / 2 / jac[:, None])[..., None]
        self.d, self.lift = t(E.d), t(E.lift)
        self.match(mesh, fv.mean(2))
        self.c = inp.get("c")
        self.eps, self.mu = inp.get("eps"), inp.get("mu")
        self.x = inp["x"]
        self.given = t(_inflow(self.x.cpu().numpy())) if case["bc"] == "given" else None

    def match(self, mesh, centre):
        """Each face node's own and opposite volume node; boundary kinds."""
        E, dim, K, nf = self.E, self.case["dim"], self.K, self.nf
        ids = np.arange(len(mesh.points))
        if self.case["bc"] == "periodic":
            nx, ny = self.case["n"] + 1, self.case["m"] + 1
            ids = (ids // nx) % (ny - 1) * nx + (ids % nx) % (nx - 1)
        fid = ids[mesh.elements][:, _FACES[dim]]                   # [K, nf, dim]
        rank = np.argsort(fid, axis=2)
        own = np.arange(K)[:, None, None] * self.Np + E.fnodes[None]
        canon = np.empty_like(own)
        for f in range(nf):
            for perm in itertools.permutations(range(dim)):
                sel = np.all(rank[:, f] == perm, axis=1)
                canon[sel, f] = E.canon[f, perm]
        flat = np.sort(fid, axis=2).reshape(K * nf, dim)
        order = np.lexsort(flat.T)
        same = np.all(flat[order][1:] == flat[order][:-1], axis=1)
        p, q = order[:-1][same], order[1:][same]
        other = np.full(K * nf, -1)
        other[p], other[q] = q, p
        own2, canon2 = own.reshape(K * nf, -1), canon.reshape(K * nf, -1)
        ext = own2.copy()
        inner = np.nonzero(other >= 0)[0]
        in_order = np.take_along_axis(own2[other[inner]], canon2[other[inner]], 1)
        e = np.empty_like(in_order)
        np.put_along_axis(e, canon2[inner], in_order, 1)
        ext[inner] = e
        self.own, self.ext = self.t(own), self.t(ext.reshape(own.shape))
        bdry = (other < 0).reshape(K, nf)
        self.bdry = self.t(bdry)[..., None]
        self.open = self.t(bdry & (np.abs(centre[..., 0] - 1) < 1e-9))[..., None]
        self.inflow = self.t(bdry & np.any(np.abs(centre + 1) < 1e-9, axis=-1))[..., None]

    def grad(self, w):
        """[dim][F, K, Np] physical derivatives of [F, K, Np]."""
        dr = torch.einsum("rij,fkj->rfki", self.d, w)
        return torch.einsum("krx,rfki->xfki", self.inv, dr)

    def lifted(self, flux):
        fl = torch.stack(flux) * self.fscale
        return fl.reshape(fl.shape[0], self.K, -1) @ self.lift.T

    def __call__(self, w, c=None, source=None):
        """w [F, K*Np] -> [F, K*Np]"""
        model, flux = self.case["model"], self.case["flux"]
        dim, n = self.case["dim"], self.n
        shape = w.shape
        m, p = w[:, self.own], w[:, self.ext]                      # [F, K, nf, Nfp]
        bd, op = self.bdry, self.open & (self.case["bc"] == "open")
        wv = w.reshape(shape[0], self.K, self.Np)
        dot = lambda a, b: sum(x * y for x, y in zip(a, b))        # noqa: E731
        if model == "varadv":
            return self.varadv(w[0]).reshape(shape)
        g = self.grad(wv)
        if model == "advection":
            v = _advection_v(dim)
            nv = dot(n, v)
            up = torch.where(bd, self.given[self.own], p[0]) if self.given is not None else p[0]
            um = m[0]
            if flux == "upwind":
                weak = nv * torch.where(nv > 0, um, up)
            else:
                weak = 0.5 * (um + up) * nv
                if flux == "lf":
                    weak = weak + 0.5 * float(np.linalg.norm(v)) * (um - up)
            f = um * nv - weak
            f = torch.where(bd & ~self.inflow, torch.zeros_like(f), f)
            return (self.lifted([f]) - sum(v[x] * g[x] for x in range(dim))).reshape(shape)
        if model in ("wave", "varwave"):
            um, vm = m[0], list(m[1:])
            nvm = dot(n, vm)
            up = torch.where(op, 0.5 * (um - nvm), torch.where(bd, -um, p[0]))
            vp = [torch.where(op, 0.5 * n[x] * (nvm - um), torch.where(bd, vm[x], p[1 + x]))
                  for x in range(dim)]
            if model == "wave":
                s = 1.0 if flux == "upwind" else 0.0
                w0 = 0.5 * (nvm + dot(n, vp)) - s * 0.5 * (um - up)
                jump = dot(n, [a - b for a, b in zip(vm, vp)])
                f = [w0 - nvm] + [0.5 * (um + up) * n[x] - s * 0.5 * n[x] * jump - um * n[x]
                                  for x in range(dim)]
                vol = torch.stack([sum(g[x][1 + x] for x in range(dim))]
                                  + [g[x][0] for x in range(dim)])
            else:
                c = self.c if c is None else c
                cm, cp = c[self.own], c[self.ext]
                s = 1.0 if flux == "upwind" else 0.0
                du = cp * up - cm * um
                dv = cp * dot(n, vp) - cm * nvm
                f = [0.5 * dv + s * du] + [(0.5 * du + s * dv) * n[x] for x in range(dim)]
                cv = c.reshape(self.K, self.Np)
                div = cv * sum(g[x][1 + x] for x in range(dim))
                if source is not None:
                    div = div - source.reshape(self.K, self.Np)
                vol = torch.stack([div] + [cv * g[x][0] for x in range(dim)])
            return (vol + self.lifted(f)).reshape(shape)
        return self.maxwell(m, p, g, bd, op).reshape(shape)

    def maxwell(self, m, p, g, bd, op):
        model, flux = self.case["model"], self.case["flux"]
        slots = {"tm": [2, 3, 4], "te": [0, 1, 5]}.get(model, list(range(6)))
        zero = torch.zeros_like(m[0])

        def six(x, z):
            return [x[slots.index(s)] if s in slots else z for s in range(6)]

        m, p = six(m, zero), six(p, zero)
        n = [x.expand_as(zero) for x in self.n] + [zero] * (3 - len(self.n))
        zm = zp = torch.ones((), dtype=zero.dtype, device=zero.device)
        if model == "material":
            z = torch.sqrt(self.mu / self.eps)
            zm, zp = z[self.own], z[self.ext]
        e, h = m[:3], m[3:]
        ne, nh = _cross(n, e), _cross(n, h)
        nne, nnh = _cross(n, ne), _cross(n, nh)
        out = []
        for k in range(3):
            out.append(torch.where(op, e[k] + 0.5 * (nne[k] - zm * nh[k]),
                                   torch.where(bd, -e[k], p[k])))
        for k in range(3):
            out.append(torch.where(op, h[k] + 0.5 * (nnh[k] + ne[k] / zm),
                                   torch.where(bd, h[k], p[3 + k])))
        de, dh = [m[k] - out[k] for k in range(3)], [m[3 + k] - out[3 + k] for k in range(3)]
        if flux == "lf":
            f = [-0.5 * x for x in _cross(n, dh)] + [0.5 * x for x in _cross(n, de)]
        else:
            al = 1.0 if flux == "upwind" else 0.0
            nde, ndh = _cross(n, de), _cross(n, dh)
            fe = _cross(n, [zp * dh[k] - al * nde[k] for k in range(3)])
            fh = _cross(n, [de[k] / zp + al * ndh[k] for k in range(3)])
            f = [-x / (zm + zp) for x in fe] + [x / (1 / zm + 1 / zp) for x in fh]
        vz = torch.zeros_like(g[0][0])
        gs = [six(g[x], vz) for x in range(len(self.n))] + [[vz] * 6] * (3 - len(self.n))
        vol = [gs[1][5] - gs[2][4], gs[2][3] - gs[0][5], gs[0][4] - gs[1][3],
               gs[2][1] - gs[1][2], gs[0][2] - gs[2][0], gs[1][0] - gs[0][1]]
        r = torch.stack([vol[s] for s in slots]) + self.lifted([f[s] for s in slots])
        if model == "material":
            div = [self.eps if s < 3 else self.mu for s in slots]
            r = r / torch.stack(div).reshape(r.shape)
        return r

    def varadv(self, u):
        """Weak form; Gauss points on the faces as the rule of degree 3N."""
        E, t, dim, order = self.E, self.t, 2, self.case["order"]
        q, wq = _gauss_simplex(dim, (3 * order) // 2 + 2)
        phi = t(E.phi(q))
        v = [-self.x[:, 1], self.x[:, 0]]
        uq = u.reshape(self.K, self.Np) @ phi.T
        vq = [x.reshape(self.K, self.Np) @ phi.T for x in v]
        r = 0.0
        for a in range(dim):
            proj = t(E.minv @ (E.phi(q, a).T * wq))
            r = r + (uq * sum(self.inv[:, a, x, None] * vq[x] for x in range(dim))) @ proj.T
        gx, gw = np.polynomial.legendre.leggauss((3 * order) // 2 + 1)
        vert = np.concatenate([-np.ones((1, dim)), 2 * np.eye(dim) - 1])
        up = torch.where(self.bdry, self.given[self.own], u[self.ext])
        cmax = (v[0] ** 2 + v[1] ** 2).reshape(self.K, self.Np).amax(1)
        for f, (i, j) in enumerate(_FACES[dim]):
            pts = vert[i] + (vert[j] - vert[i]) * (gx[:, None] + 1) / 2
            full = E.phi(pts)
            trace = t(full[:, E.fnodes[f]])
            own = self.own[:, f]
            n = [x[:, f] for x in self.n]
            uM, uP = u[own] @ trace.T, up[:, f] @ trace.T
            vf = [x[own] @ trace.T for x in v]
            nv = sum(n[x] * vf[x] for x in range(dim))
            if self.case["flux"] == "upwind":
                fl = nv * torch.where(nv > 0, uM, uP)
            else:
                fl = 0.5 * nv * (uM + uP)
                if self.case["flux"] == "lf":
                    nb = torch.div(self.ext[:, f, 0], self.Np, rounding_mode="floor")
                    fl = fl - 0.5 * (uP - uM) * torch.maximum(cmax, cmax[nb])[:, None]
            r = r - (fl * self.fscale[:, f]) @ t(E.minv @ (full.T * gw)).T
        return r

    def step(self, w, dt, t0=0.0, c=None, source=None):
        res = torch.zeros_like(w)
        for a, b, cs in zip(_LSRK_A, _LSRK_B, _LSRK_C):
            src = None if source is None else source * _amplitude(t0 + cs * dt)
            res = a * res + dt * self(w, c, src)
            w = w + b * res
        return w


def exact(case, seed):
    if case["kind"] == "ensemble":
        out = []
        for c, s in _members(case, seed):
            inp = _inputs(c, s)
            out.append(_Plain(c, inp).step(inp["w"].double(), _time_step(c)))
        return out
    inp = _inputs(case, seed)
    plain, w, dt = _Plain(case, inp), inp["w"].double(), _time_step(case)
    if case["kind"] == "rhs":
        r = plain(w)
        return r[0] if len(r) == 1 else r
    if case["kind"] == "step":
        return plain.step(w, dt)
    if case["kind"] == "loop":
        for _ in range(case["steps"]):
            w = plain.step(w, dt)
        E = plain.E
        jac = torch.as_tensor(np.abs(np.linalg.det(_maps(inp["mesh"])[1])), device=w.device)
        mass = torch.as_tensor(E.vinv.T @ E.vinv, device=w.device)
        wv = w.reshape(len(w), plain.K, plain.Np)
        return w, float(torch.einsum("fki,ij,fkj,k->", wv, mass, wv, jac).sqrt())
    w.requires_grad_(True)
    c = inp["c"].requires_grad_(True) if "c" in inp else None
    wrt = [w] if c is None else [w, c]
    if case["kind"] == "grad":
        out = plain(w, c)
        return [out.detach(), *torch.autograd.grad(out, wrt, inp["lam"])]
    # traces
    E, v = plain.E, inp["mesh"].points[inp["mesh"].elements]
    inv, (_, _, b) = plain.inv.cpu().numpy(), _maps(inp["mesh"])
    rows = []
    for pt in inp["points"]:
        r = np.einsum("kij,kj->ki", inv, pt - b)
        el = int(np.nonzero(np.all(r >= -1, axis=1) & (r.sum(1) <= 0))[0][0])
        rows.append((el, torch.as_tensor(E.phi(r[el][None])[0], device=w.device)))

    def receive(q):
        return torch.stack([q[0, el * plain.Np:(el + 1) * plain.Np] @ ph for el, ph in rows])

    q, t, traces = w, 0.0, [receive(w)]
    for _ in range(case["steps"]):
        q = plain.step(q, dt, t, c, inp["source"])
        t += dt
        traces.append(receive(q))
    traces = torch.stack(traces)
    return [traces.detach(), *torch.autograd.grad((traces * traces).sum(), wrt)]

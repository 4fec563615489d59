"""The workloads this library's performance is followed on.

A case is a dict of plain values; `listed()` gives the fixed ones and `draw()`
further ones of the same ranges.  Every case goes through the package's public
entry points, as a program that uses it does:

  solve      SetSolution, ForwardStep over some RK3 steps and (where "entropy"
             is set) the entropy that SELF's ForwardStep reports at the end of
             each output interval; any model, degree, form and shock closure
  tendency   SetSolution and CalculateTendency (callers with their own time
             integrator)
  ensemble   uneven ShallowWater instances advanced together
  operators  one CompressibleIdealGas2D tendency and RK update through the
             operator-by-operator entry points, in the order of SELF's own
             CalculateTendency: what a SELF program that is merely relinked
             against the library calls
  fields     SELF's field classes: BR1 gradient, divergence, interpolation to
             the plot grid and the integral of a field
  learn      the closure MLP: features of a state, training, inference

`exact()` restates each in plain 64-bit torch on the same structured meshes.
"""
import math

import numpy as np
import torch

import self_b200 as S
from self_b200 import closure as C
from self_b200 import ensemble as E

GAMMA = 1.4
FORMS = {"fp64": S.FP64, "fp32": S.FP32_BULK, "ref": S.FP64_REF}
NV = {"lsw": 3, "sw": 3, "cig": 4}
RK_A = (0.0, -5.0 / 9.0, -153.0 / 128.0)
RK_G = (1.0 / 3.0, 15.0 / 16.0, 8.0 / 15.0)


# --------------------------------------------------------------------- cases
def _solve(name, model, form, N, nx, ny, steps, walls=False, closure="off", entropy=False, perturb=0.0, sources=False):
    case = {"kind": "solve", "model": model, "form": form, "N": N, "nx": nx, "ny": ny, "steps": steps, "walls": walls,
            "closure": closure, "entropy": entropy, "perturb": perturb, "sources": sources}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the reference's gravity-wave release on its 10x10 block: launches and latency are all there is
        _solve("lsw_10x10_n7", "lsw", "fp64", 7, 10, 10, 20, walls=True, entropy=True),
        # a mesh of about a thousand elements, the size of the reference's own examples, with gravity and drag
        _solve("cig_36x28_n7", "cig", "fp64", 7, 36, 28, 10, walls=True, sources=True, entropy=True),
        # the headline solve (density wave, 128x128, degree 7), a stretch of its 200 steps
        _solve("cig_128x128_n7", "cig", "fp64", 7, 128, 128, 10, perturb=0.02),
        # an even degree (an odd number of nodes), walls and topography, a ragged mesh
        _solve("sw_151x93_n4", "sw", "fp64", 4, 151, 93, 10, walls=True, sources=True, entropy=True),
        # a large solve in the FP32-bulk form: 67 million degrees of freedom
        _solve("cig_512x512_n7_fp32", "cig", "fp32", 7, 512, 512, 3, perturb=0.02),
        # the Riemann problem with the learned closure in the FP32-bulk form
        _solve("cig_256x256_n5_mlp", "cig", "fp32", 5, 256, 256, 4, closure="mlp"),
        # a shock band with the indicator closure, double precision, reported like an output interval
        _solve("cig_120x88_n7_shock", "cig", "fp64", 7, 120, 88, 5, closure="indicator", entropy=True, perturb=0.02),
        # the tendency alone with the reference's roundings, as a caller with its own integrator asks for it
        {"name": "tendency_ref_96x80_n7", "kind": "tendency", "model": "cig", "form": "ref", "N": 7, "nx": 96,
         "ny": 80, "walls": True, "perturb": 0.0, "sources": True},
        # uneven batched ShallowWater members of degrees 3, 5 and 7
        {"name": "ensemble_64_fp32", "kind": "ensemble", "form": "fp32", "members": 64, "most": 64, "steps": 5},
        # an unmodified SELF tendency, operator by operator
        {"name": "operators_64x64_n7", "kind": "operators", "N": 7, "nx": 64, "ny": 64},
        # field classes on a mesh of the reference's GeophysicalBlock2DMedium kind
        {"name": "fields_100x75_n3", "kind": "fields", "N": 3, "M": 7, "nVar": 5, "nx": 100, "ny": 75},
        # learning the closure from the states of a 128x128 run
        {"name": "learn_16384_n7", "kind": "learn", "N": 7, "n": 16384, "batch": 4096, "epochs": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["tendency", "ensemble", "operators", "fields", "learn"])
    if kind in ("solve", "tendency"):
        model = rng.choice(["lsw", "sw", "cig", "cig"])
        N = rng.choice([2, 3, 4, 5, 6, 7, 7])
        most = 220 if kind == "solve" else 160
        nx, ny = _log_int(rng, 8, most), _log_int(rng, 8, most)
        walls = rng.random() < 0.5
        perturb = rng.choice([0.0, 0.02])
        sources = rng.random() < 0.5
        if kind == "tendency":
            return {"kind": kind, "model": model, "form": rng.choice(["fp64", "ref"]), "N": N, "nx": nx, "ny": ny,
                    "walls": walls, "perturb": perturb, "sources": sources}
        closure = rng.choice(["off", "indicator", "mlp"]) if model == "cig" and N >= 5 and not walls else "off"
        return _solve(None, model, rng.choice(["fp64", "fp64", "fp32", "ref"]), N, nx, ny, rng.randint(3, 10),
                      walls=walls, closure=closure, entropy=rng.random() < 0.5, perturb=perturb,
                      sources=sources and closure == "off")
    if kind == "ensemble":
        return {"kind": kind, "form": rng.choice(["fp64", "fp32"]), "members": _log_int(rng, 8, 80),
                "most": rng.choice([24, 40, 64]), "steps": rng.randint(2, 6)}
    if kind == "operators":
        return {"kind": kind, "N": rng.choice([2, 3, 4, 5, 6, 7]), "nx": _log_int(rng, 10, 120),
                "ny": _log_int(rng, 10, 120)}
    if kind == "fields":
        return {"kind": kind, "N": rng.choice([2, 3, 4, 5, 6, 7]), "M": rng.choice([3, 5, 7, 10]),
                "nVar": rng.randint(1, 6), "nx": _log_int(rng, 10, 120), "ny": _log_int(rng, 10, 120)}
    return {"kind": kind, "N": rng.choice([5, 6, 7]), "n": _log_int(rng, 3000, 40000),
            "batch": rng.choice([1000, 4096, 8192]), "epochs": rng.randint(1, 2)}


# -------------------------------------------------------------- inputs of a seed
def _rng(seed, salt=0):
    return np.random.Generator(np.random.PCG64([int(seed), salt]))


def _dt(case):
    """A CFL-0.4 step for signal speeds up to 2.2; a tenth of it under the closure (its explicit viscous limit)."""
    h = min(1.0 / case["nx"], 1.0 / case["ny"])
    return (0.04 if case.get("closure", "off") != "off" else 0.4) * h / case["N"] ** 2 / 2.2


def _wave(X, Y, r):
    """A few seeded long waves of unit size, periodic on [0, 1]^2."""
    f = torch.zeros_like(X)
    for _ in range(3):
        kx, ky = int(r.integers(1, 3)), int(r.integers(1, 3))
        f = f + torch.sin(2 * np.pi * kx * X + r.uniform(0, 6.28)) * torch.sin(2 * np.pi * ky * Y + r.uniform(0, 6.28))
    return f / 3.0


def _topography(X, Y):
    h = torch.ones_like(X)
    for a, s, cx, cy in ((0.15, 0.12, 0.3, 0.4), (0.1, 0.2, 0.7, 0.6)):
        h = h - a * torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / s ** 2)
    return h


def _gas(rho, u, v, p):
    return torch.stack([rho * u, rho * v, rho, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], dim=1)


def _initial(case, X, Y, seed):
    """(nEl, nVar, P, P) state of the seed on node coordinates X, Y (nEl, P, P)."""
    r = _rng(seed)
    if case["model"] == "lsw":
        cx, cy, a = r.uniform(0.35, 0.65), r.uniform(0.35, 0.65), r.uniform(0.005, 0.015)
        eta = a * torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / 0.01)
        return torch.stack([0.01 * _wave(X, Y, r), 0.01 * _wave(X, Y, r), eta], dim=1)
    if case["model"] == "sw":
        h = _topography(X, Y) if case["sources"] else torch.ones_like(X)
        H = h + r.uniform(0.002, 0.01) * torch.exp(-((X - 0.4) ** 2 + (Y - 0.55) ** 2) / 0.01)
        return torch.stack([0.01 * _wave(X, Y, r), 0.01 * _wave(X, Y, r), H], dim=1)
    one = torch.ones_like(X)
    if case.get("closure", "off") == "off":
        rho = 1.0 + 0.1 * _wave(X, Y, r)
        return _gas(rho, 0.5 * one + 0.05 * _wave(X, Y, r), 0.3 * one, one + 0.02 * _wave(X, Y, r))
    # a smooth wave and, across seeded lines, a shock tube band
    rho = 1.0 + 0.1 * _wave(X, Y, r)
    x0, y0 = r.uniform(0.3, 0.7, 2)
    band, left = (Y - y0).abs() < 0.05, X < x0
    rho = torch.where(band, torch.where(left, one, 0.125 * one), rho)
    p = torch.where(band, torch.where(left, one, 0.1 * one), one)
    return _gas(rho, torch.where(band, 0 * one, 0.5 * one), torch.where(band, 0 * one, 0.3 * one), p)


def _mlp(N):
    """A closure network whose output follows the indicator's ramp (its first unit reads the density's top shell);
    the other units hold small fixed weights that are evaluated with it."""
    mlp = C.ClosureMLP(seed=7)
    W1, b1, W2, b2, w3, _ = mlp.unpack()
    W1[0], W2[0], w3[:] = 0.0, 0.0, 0.0
    W1[0, 5], W2[0, 0], w3[0] = 1.0, 1.0, 4.0
    b1[0], b2[0] = -(7.0 - 4.0 * math.log10(N)) / 8.0, 0.0
    return mlp


def _modal_states(N, n, seed, device):
    """(n, 4, P, P) gas states whose Legendre modes decay at seeded rates, from resolved to rough."""
    P = N + 1
    r = _rng(seed, 3)
    x, _ = np.polynomial.legendre.leggauss(P)
    V = np.polynomial.legendre.legvander(x, N) * np.sqrt(np.arange(P) + 0.5)
    k = np.maximum(np.arange(P)[:, None], np.arange(P)[None, :])
    decay = 10.0 ** (-r.uniform(0.15, 0.9, (n, 1, 1)) * k) * (k > 0)
    V = torch.as_tensor(V, device=device)

    def field(scale, mean):
        c = torch.as_tensor(scale * decay * r.uniform(-1, 1, (n, P, P)), device=device)
        return mean + torch.einsum("ik,ekl,jl->eji", V, c, V)

    rho = field(0.2, 1.0)
    one = torch.ones_like(rho)
    return _gas(rho, 0.3 * one, 0.1 * one, field(0.1, 1.0))


def _members(case, seed):
    """Ensemble members: the sizes are the case's, topography and wave the seed's."""
    inst = E.make_instances(case["members"], seed=0, nmax=case["most"])
    new = E.make_instances(case["members"], seed=int(seed) + 1, nmax=case["most"])
    for a, b in zip(inst, new):
        a.bumps, a.wave = b.bumps, b.wave
    return inst


def _mesh(case):
    walls = case["walls"]
    return S.Mesh2D(case["nx"], case["ny"], periodic=(not walls, not walls), perturbation=case["perturb"],
                    bcid=S.BC_NONORMALFLOW)


def _model(case, seed):
    mesh = _mesh(case)
    geo = S.SEMQuad(S.Lagrange(case["N"], S.GAUSS, case["N"], S.UNIFORM), mesh)
    X, Y = geo.x[:, 0, :, :, 0], geo.x[:, 0, :, :, 1]
    form = FORMS[case["form"]]
    if case["model"] == "lsw":
        m = S.LinearShallowWater(mesh, geo, form=form)
        m.SetBathymetry(_topography(X, Y).unsqueeze(1) if case["sources"] else 1.0)
        m.SetCoriolis((0.5 + Y).unsqueeze(1))
    elif case["model"] == "sw":
        m = S.ShallowWater(mesh, geo, form=form)
        if case["sources"]:
            m.SetTopography(_topography(X, Y).unsqueeze(1))
    else:
        m = S.CompressibleIdealGas2D(mesh, geo, form=form)
        if case["sources"]:
            m.SetGravity((0.1 * Y).unsqueeze(1))
            m.SetDrag(0.01)
    q0 = _initial(case, X, Y, seed)
    m.SetSolution(q0)
    if case.get("closure", "off") != "off":
        mlp = case["closure"] == "mlp"
        m.SetClosure(S.CLOSURE_MLP if mlp else S.CLOSURE_INDICATOR, mlp=_mlp(case["N"]) if mlp else None)
    return m, q0


def _zeros(*shape):
    return torch.zeros(shape, device="cuda", dtype=torch.float64)


def _operator_calls(s):
    """One CalculateTendency and UpdateGRK of SELF_CompressibleIdealGas2D by the drop-in entry points: (call, arguments)
    with the pointers that a Fortran program keeps in its c_ptr variables."""
    L, w = s["geo"].interp, S.lib()
    N, n, geo, mesh = L.N, s["n"], s["geo"], s["mesh"]

    def p(t):
        return S._lib.pp(t.data_ptr())

    bM, dgM, qw = p(L.device("bMatrix")), p(L.device("dgMatrix")), p(L.device("qWeights"))
    nh, ns, si, rank = p(geo.nHat), p(geo.nScale), p(mesh.sideInfo_d), p(s["rank"])
    a = {k: p(v) for k, v in s.items() if isinstance(v, torch.Tensor)}
    calls = [(w.CalculateDiagnostics_CompressibleIdealGas2D_gpu_wrapper, (a["q"], a["diag"], GAMMA, 1.0, N, 4, 4, n)),
             (w.ConservativeToPrimitive_CompressibleIdealGas2D_gpu_wrapper, (a["q"], a["prim"], GAMMA, N, 4, n))]
    for f, b, x in (("q", "qb", "qx"), ("prim", "pb", "px"), ("diag", "db", "dx")):
        calls += [(w.ScalarBoundaryInterp_2D_gpu_wrapper, (bM, a[f], a[b], N, 4, n)),
                  (w.SideExchange_MappedScalar2D_gpu_wrapper, (a[x], a[b], si, rank, 0, 0, N, 4, n))]
    calls += [
        (w.SetBoundaryCondition_CompressibleIdealGas2D_gpu_wrapper,
         (a["qb"], a["qx"], a["qp"], a["pb"], a["px"], a["pp"], a["db"], a["dx"], a["dp"], nh, si, N, 4, 4, n)),
        (w.Source_CompressibleIdealGas2D_gpu_wrapper, (a["src"], a["q"], a["env"], N, 4, n)),
        (w.NaiveLLF_CompressibleIdealGas2D_gpu_wrapper,
         (a["fb"], a["qb"], a["qx"], a["pb"], a["px"], a["db"], a["dx"], nh, ns, N, 4, 4, n)),
        (w.Flux_CompressibleIdealGas2D_gpu_wrapper, (a["flux"], a["q"], a["prim"], N, 4, n)),
        (w.ContravariantProjection_MappedVector2D_gpu_wrapper, (a["flux"], p(geo.dsdx), N, 4, n)),
        (w.VectorDGDivergence_2D_gpu_wrapper, (dgM, bM, qw, a["flux"], a["fb"], a["div"], N, 4, n)),
        (w.JacobianWeight_MappedScalar2D_gpu_wrapper, (a["div"], p(geo.J), N, 4, n)),
        (w.CalculateDSDt_Model2D_gpu_wrapper, (a["div"], a["src"], a["dSdt"], N, 4, n)),
        (w.UpdateGRK_Model2D_gpu_wrapper, (a["G"], a["q"], a["dSdt"], RK_A[0], RK_G[0], s["dt"], 4, N, 4, n))]
    return calls


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("solve", "tendency"):
        st["model"], st["q0"] = _model(case, seed)
        st["dt"] = _dt(case)
    elif kind == "ensemble":
        st["inst"] = _members(case, seed)
        st["ens"] = E.ShallowWaterEnsemble(st["inst"], form=FORMS[case["form"]], autotune=False)
    elif kind == "operators":
        N, P = case["N"], case["N"] + 1
        c = dict(case, walls=True, perturb=0.02, model="cig", sources=True)
        mesh = _mesh(c)
        geo = S.SEMQuad(S.Lagrange(N, S.GAUSS, N, S.UNIFORM), mesh)
        X, Y = geo.x[:, 0, :, :, 0], geo.x[:, 0, :, :, 1]
        n = mesh.nElem
        env = S.MappedScalar2D(geo.interp, 2, n)
        env.interior[:, 0] = 0.1 * Y
        g = S.MappedVector2D(geo.interp, 2, n)
        env.GradientSF(geo, g)
        st.update(mesh=mesh, geo=geo, dt=_dt(dict(case)), q0=_initial(c, X, Y, seed), env=g.interior, n=n)
        st["rank"] = torch.zeros(n, device="cuda", dtype=torch.int32)
        for k in ("q", "prim", "diag", "src", "div", "dSdt", "G"):
            st[k] = _zeros(n, 4, P, P)
        st["flux"] = _zeros(n, 4, P, P, 2)
        for k in ("qb", "qx", "qp", "pb", "px", "pp", "db", "dx", "dp", "fb"):
            st[k] = _zeros(n, 4, 4, P)
        st["calls"] = _operator_calls(st)
    elif kind == "fields":
        N, nVar = case["N"], case["nVar"]
        c = dict(case, walls=False, perturb=0.02)
        mesh = _mesh(c)
        interp = S.Lagrange(N, S.GAUSS, N, S.UNIFORM)
        geo = S.SEMQuad(interp, mesh)
        r = _rng(seed, 1)
        X, Y = geo.x[:, 0, :, :, 0], geo.x[:, 0, :, :, 1]
        f = S.MappedScalar2D(interp, nVar, mesh.nElem)
        for v in range(nVar):
            f.interior[:, v] = 1.0 + _wave(X, Y, r)
        grad = S.MappedVector2D(interp, nVar, mesh.nElem)
        grad.boundaryNormal.copy_(torch.as_tensor(0.01 * r.standard_normal((1, 4, nVar, N + 1)), device="cuda"))
        plot = S.Lagrange(N, S.GAUSS, case["M"], S.UNIFORM)
        fp = S.MappedScalar2D(plot, nVar, mesh.nElem)  # the field on its plot grid's interpolant
        out = S.MappedScalar2D(S.Lagrange(case["M"], S.GAUSS, case["M"], S.UNIFORM), nVar, mesh.nElem)
        fp.interior = f.interior
        st.update(mesh=mesh, geo=geo, f=f, grad=grad, div=S.MappedScalar2D(interp, nVar, mesh.nElem), fp=fp, out=out)
    else:
        st["interp"] = S.Lagrange(case["N"], S.GAUSS, case["N"], S.UNIFORM)
        st["q"] = _modal_states(case["N"], case["n"], seed, "cuda")
    return st


# ------------------------------------------------------------------- one pass
def _operators(s):
    for call, args in s["calls"]:
        call(*args)
    return {"dSdt": s["dSdt"], "q": s["q"]}


def _fields(s):
    f, g = s["f"], s["grad"]
    f.BoundaryInterp()
    f.SideExchange(s["mesh"])
    f.BassiRebaySides()
    f.GradientBR(s["geo"], g)
    g.BoundaryInterp()
    g.SideExchange(s["mesh"])
    out = {"gradient boundary": g.boundary, "gradient ext": g.extBoundary}
    g.ContravariantProjection(s["geo"])
    g.Divergence(s["geo"], s["div"])
    s["fp"].GridInterp(s["out"])
    out.update(divergence=s["div"].interior, plot=s["out"].interior, integral=f.Integral(s["geo"], 1))
    return out


def _learn(s):
    c = s["case"]
    act, feat = C.features(s["q"], s["interp"])
    mlp = C.ClosureMLP(seed=1)
    loss = mlp.train(feat, act, epochs=c["epochs"], batch=c["batch"], lr=2e-3, seed=1)
    return {"activation": act, "features": feat, "parameters": mlp.params, "loss": loss, "output": mlp.infer(feat)}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        m = st["model"]
        m.SetSolution(st["q0"])
        m.ForwardStep(case["steps"], st["dt"])
        out = {"solution": m.solution}
        if case["entropy"]:
            out["entropy"] = m.CalculateEntropy()
        return out
    if kind == "tendency":
        st["model"].SetSolution(st["q0"])
        return {"dSdt": st["model"].CalculateTendency()}
    if kind == "ensemble":
        st["ens"].reset()
        st["ens"].ForwardStep(case["steps"])
        for h in st["ens"].handles.values():
            torch.cuda.current_stream().wait_stream(h["stream"])
        return {"N%d" % N: h["model"].solution for N, h in st["ens"].handles.items()}
    if kind == "operators":
        st["q"].copy_(st["q0"])
        return _operators(st)
    return _fields(st) if kind == "fields" else _learn(st)


# ----------------------------------------------------- what a pass has to move
def _stage_work(model, form, N, nEl):
    """One RK stage: solution and register read and written, metric terms, connectivity and the neighbours' states read."""
    P, nv = N + 1, NV[model]
    reg = 4 if form == "fp32" else 8
    nbytes = 16 * nv * P * P + 2 * reg * nv * P * P + 8 * 4 * nv * P + 8 * (5 * P * P + 12 * P) + 80
    flops = nv * P * P * (4 * P + 30) + 4 * P * 60 + (9 if model == "cig" else nv) * 8 * P * P
    return {"bytes": nbytes * nEl, "flops": flops * nEl}


def work(case):
    kind = case["kind"]
    if kind in ("solve", "tendency"):
        nEl = case["nx"] * case["ny"]
        w = _stage_work(case["model"], case["form"], case["N"], nEl)
        k = 3 * case["steps"] if kind == "solve" else 1
        return {"bytes": k * w["bytes"], "flops": k * w["flops"]}
    if kind == "ensemble":
        tot = {"bytes": 0, "flops": 0}
        for i in E.make_instances(case["members"], seed=0, nmax=case["most"]):
            w = _stage_work("sw", case["form"], i.N, i.nElem)
            for k in tot:
                tot[k] += 3 * case["steps"] * w[k]
        return tot
    if kind == "operators":
        P, nEl = case["N"] + 1, case["nx"] * case["ny"]
        # every operator reads its inputs and writes its outputs once: node and face values of four variables
        node, face = 32 * P * P, 32 * 4 * P
        nbytes = node * 30 + face * 26 + 8 * (10 * P * P + 24 * P) + 400
        return {"bytes": nbytes * nEl, "flops": nEl * 4 * P * P * (10 * P + 60)}
    if kind == "fields":
        P, Q, nEl, nv = case["N"] + 1, case["M"] + 1, case["nx"] * case["ny"], case["nVar"]
        node, face = 8 * nv * P * P, 8 * nv * 4 * P
        nbytes = node * 15 + face * 17 + 8 * nv * Q * Q + 8 * (12 * P * P + 12 * P) + 160
        return {"bytes": nbytes * nEl, "flops": nEl * nv * (P * P * (20 * P + 40) + 2 * Q * P * (P + Q))}
    n, steps = case["n"], case["epochs"] * -(-case["n"] // case["batch"])
    per = 36 * 32 + 32 * 32 + 32
    P = case["N"] + 1
    return {"bytes": n * (16 * P * P + 4 * 37 * 2) + steps * case["batch"] * 148,
            "flops": n * (8 * P ** 3 + 2 * per) + steps * case["batch"] * 6 * per}


# ------------------------------------------- the same in plain 64-bit torch
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Grid:
    """Gauss operators and metric terms of the structured mesh; arrays are (nEl, ..., j, i), faces (S, E, N, W)."""

    def __init__(self, N, nx, ny, walls, perturb):
        P = N + 1
        self.N, self.nx, self.ny, self.walls = N, nx, ny, walls
        x, w = np.polynomial.legendre.leggauss(P)
        if P == 4:  # the reference's Newton iteration finds the inner pair in this order
            x[1], x[2] = x[2], x[1]
        bw = np.array([1.0 / np.prod([x[i] - x[j] for j in range(P) if j != i]) for i in range(P)])
        D = np.array([[0.0 if i == j else bw[j] / bw[i] / (x[i] - x[j]) for j in range(P)] for i in range(P)])
        D[np.arange(P), np.arange(P)] = -D.sum(axis=1)

        def basis(t):
            return np.array([np.prod([(t - x[j]) / (x[i] - x[j]) for j in range(P) if j != i]) for i in range(P)])

        dev = dict(device=_device(), dtype=torch.float64)
        self.dev, self.xi = dev, x
        self.basis = basis
        t = lambda a: torch.as_tensor(a, **dev)  # noqa: E731
        self.w, self.D = t(w), t(D)
        self.W = t(-(w[:, None] * D / w[None, :]).T)  # weak derivative: W[i, m]
        self.lo, self.hi = t(basis(-1.0)), t(basis(1.0))
        gx, gy = np.meshgrid(np.arange(nx + 1) / nx, np.arange(ny + 1) / ny)
        if perturb:
            d = perturb * min(1.0 / nx, 1.0 / ny) * np.sin(2 * np.pi * gx) * np.sin(2 * np.pi * gy)
            d[0], d[-1], d[:, 0], d[:, -1] = 0, 0, 0, 0
            gx, gy = gx + d, gy + d
        a, b = t((1 - x) / 2), t((1 + x) / 2)

        def bil(g):
            c = [t(v.reshape(-1)) for v in (g[:-1, :-1], g[:-1, 1:], g[1:, :-1], g[1:, 1:])]
            o = lambda u, s: torch.einsum("e,j,i->eji", u, s[1], s[0])  # noqa: E731
            val = o(c[0], (a, a)) + o(c[1], (b, a)) + o(c[2], (a, b)) + o(c[3], (b, b))
            one = torch.ones_like(a)
            d1 = 0.5 * (o(c[1] - c[0], (one, a)) + o(c[3] - c[2], (one, b)))
            d2 = 0.5 * (o(c[2] - c[0], (a, one)) + o(c[3] - c[1], (b, one)))
            return val, d1, d2

        self.X, x1, x2 = bil(gx)
        self.Y, y1, y2 = bil(gy)
        self.J = x1 * y2 - x2 * y1
        self.m = (y2, -x2, -y1, x1)  # F1 = m0 Fx + m1 Fy, F2 = m2 Fx + m3 Fy
        mb = [self.trace(v) for v in self.m]
        self.nx_, self.ny_ = [], []
        for s, (k, sg) in enumerate(((2, -1), (0, 1), (2, 1), (0, -1))):
            self.nx_.append(sg * mb[k][s])
            self.ny_.append(sg * mb[k + 1][s])
        self.ns = [torch.sqrt(p * p + q * q) for p, q in zip(self.nx_, self.ny_)]
        self.nh = [(p / n, q / n) for p, q, n in zip(self.nx_, self.ny_, self.ns)]

    def trace(self, f):
        return [f.transpose(-1, -2) @ self.lo, f @ self.hi, f.transpose(-1, -2) @ self.hi, f @ self.lo]

    def neighbour(self, tr):
        """The neighbours' traces on each side (walls: zeros there) and the mask of physical faces."""
        out = []
        for s, (opp, ax, sh) in enumerate(((2, 0, 1), (3, 1, -1), (0, 0, -1), (1, 1, 1))):
            g = tr[opp].reshape((self.ny, self.nx) + tr[opp].shape[1:])
            out.append(torch.roll(g, sh, dims=ax).reshape(tr[opp].shape))
        return out

    def wall(self, s):
        m = torch.zeros((self.ny, self.nx), device=self.dev["device"], dtype=torch.bool)
        if self.walls:
            ((m[0], m[:, -1], m[-1], m[:, 0])[s])[...] = True
        return m.reshape(-1)

    def divergence(self, Fx, Fy, fb):
        """Weak divergence / J of (nEl, v, j, i) fluxes with outward face fluxes fb[s] (nEl, v, P)."""
        m = [v.unsqueeze(1) for v in self.m]
        return self.divergence_ref(m[0] * Fx + m[1] * Fy, m[2] * Fx + m[3] * Fy, fb)

    def divergence_ref(self, F1, F2, fb):
        d = F1 @ self.W.T + self.W @ F2
        lo, hi = self.lo / self.w, self.hi / self.w
        d = d + fb[1].unsqueeze(-1) * hi + fb[3].unsqueeze(-1) * lo
        d = d + fb[2].unsqueeze(-2) * hi[:, None] + fb[0].unsqueeze(-2) * lo[:, None]
        return d / self.J.unsqueeze(1)

    def gradient_sf(self, f):
        g = []
        for k in (0, 1):
            a, b = f * self.m[k], f * self.m[2 + k]
            g.append((a @ self.D.T + self.D @ b) / self.J)
        return g

    def gradient_br(self, f, avg):
        """(gx, gy) of (nEl, v, j, i) with averaged traces avg[s] (nEl, v, P)."""
        g = []
        zero = torch.zeros_like(f)
        for k in (0, 1):
            fb = [avg[s] * (self.nh[s][k] * self.ns[s]).unsqueeze(1) for s in range(4)]
            g.append(self.divergence(f if k == 0 else zero, f if k == 1 else zero, fb))
        return g

    def integral(self, f):
        return (f * self.J * self.w * self.w[:, None]).sum()


def _reflect(u, v, a, b):
    return (b * b - a * a) * u - 2 * a * b * v, (a * a - b * b) * v - 2 * a * b * u


class _Plain:
    """The tendency and the RK3 steps of a case."""

    def __init__(self, case, seed):
        self.case = case
        self.g = _Grid(case["N"], case["nx"], case["ny"], case["walls"], case["perturb"])
        g, src = self.g, case["sources"]
        self.model = case["model"]
        self.q = _initial(case, g.X, g.Y, seed)
        h = _topography(g.X, g.Y)
        if self.model == "lsw":
            self.H = h if src else torch.ones_like(h)
            self.Hb, self.f = g.trace(self.H), 0.5 + g.Y
        elif self.model == "sw":
            self.top = h if src else torch.zeros_like(h)
            self.dh = g.gradient_sf(self.top)
            t = g.trace(self.q)
            self.vel = [[s[:, 0] / s[:, 2], s[:, 1] / s[:, 2]] for s in t]
        else:
            self.env = g.gradient_sf(0.1 * g.Y) if src else None
        self.nu = None

    def aux(self, q):
        r = 1.0 / q[:, 2]
        u, v = q[:, 0] * r, q[:, 1] * r
        p = (GAMMA - 1) * (q[:, 3] - 0.5 * (q[:, 0] * u + q[:, 1] * v))
        return u, v, p, q[:, 3] + p, torch.sqrt(GAMMA * p * r)

    def viscosity(self, q):
        case, g = self.case, self.g
        N, P = case["N"], case["N"] + 1
        s0 = -4.0 * math.log10(N)
        feat, s = _features(q, N)
        act = _activation(s, s0)
        if case["closure"] == "mlp":
            need = s >= s0 - 2.0
            act = torch.where(need, _mlp_out(_mlp(N).params, feat.float().double()), act)
        u, v, _, _, c = self.aux(q)
        lam = (torch.sqrt(u * u + v * v) + c).amax(dim=(1, 2))
        h = torch.sqrt((g.J * g.w * g.w[:, None]).sum(dim=(1, 2)))
        return act * h / N * lam

    def tendency(self, q, first=True):
        g, case = self.g, self.case
        if self.model == "cig":
            u, v, p, rh, c = self.aux(q)
            full = torch.cat([q, torch.stack([u, v, p, rh, c], dim=1)], dim=1)
        else:
            full = q
        own = g.trace(full)
        ext = g.neighbour(own)
        if self.model == "sw":
            velx = [torch.stack(t, dim=1) for t in self.vel]
            velx = g.neighbour(velx)
        fb = []
        avg = []
        for s in range(4):
            L, X = own[s], ext[s].clone()
            a, b = g.nh[s]
            w = g.wall(s)
            if case["walls"]:
                Xw = L.clone()
                Xw[:, 0], Xw[:, 1] = _reflect(L[:, 0], L[:, 1], a, b)
                if self.model == "cig":
                    Xw[:, 4], Xw[:, 5] = _reflect(L[:, 4], L[:, 5], a, b)
                X[w] = Xw[w]
            avg.append(0.5 * (L[:, :4] + X[:, :4]))
            if self.model == "lsw":
                c = torch.sqrt(self.Hb[s])
                unL, unR = L[:, 0] * a + L[:, 1] * b, X[:, 0] * a + X[:, 1] * b
                wL, wR = 0.5 * (unL + L[:, 2] / c), 0.5 * (unR - X[:, 2] / c)
                f = torch.stack([c * (wL - wR) * a, c * (wL - wR) * b, c * c * (wL + wR)], dim=1)
            elif self.model == "sw":
                vL, vR = self.vel[s], [velx[s][:, 0].clone(), velx[s][:, 1].clone()]
                for t in vR:
                    t[w] = 0.0
                unL, unR = vL[0] * a + vL[1] * b, vR[0] * a + vR[1] * b
                cL, cR = torch.sqrt(L[:, 2]), torch.sqrt(X[:, 2])
                al = torch.maximum(torch.maximum((unL + cL).abs(), (unR + cR).abs()),
                                   torch.maximum((unL - cL).abs(), (unR - cR).abs()))

                def fl(Q, un):
                    pr = 0.5 * Q[:, 2] * Q[:, 2]
                    return torch.stack([Q[:, 0] * un + pr * a, Q[:, 1] * un + pr * b, Q[:, 0] * a + Q[:, 1] * b], dim=1)

                f = 0.5 * (fl(L, unL) + fl(X, unR) + al.unsqueeze(1) * (L - X))
            else:
                def fl(Q):
                    un = Q[:, 4] * a + Q[:, 5] * b
                    return un, torch.stack([un * Q[:, 0] + Q[:, 6] * a, un * Q[:, 1] + Q[:, 6] * b,
                                            Q[:, 0] * a + Q[:, 1] * b, un * Q[:, 7]], dim=1)

                (unL, fL), (unR, fR) = fl(L), fl(X)
                al = torch.maximum(unL.abs(), unR.abs()) + torch.maximum(L[:, 8].abs(), X[:, 8].abs())
                f = 0.5 * (fL + fR + al.unsqueeze(1) * (L[:, :4] - X[:, :4]))
            fb.append(f * g.ns[s].unsqueeze(1))
        z = torch.zeros_like(q[:, 0])
        if self.model == "lsw":
            Fx = torch.stack([q[:, 2], z, self.H * q[:, 0]], dim=1)
            Fy = torch.stack([z, q[:, 2], self.H * q[:, 1]], dim=1)
            src = torch.stack([self.f * q[:, 1], -self.f * q[:, 0], z], dim=1)
        elif self.model == "sw":
            H = q[:, 2]
            u, v, pr = q[:, 0] / H, q[:, 1] / H, 0.5 * H * H
            Fx = torch.stack([u * q[:, 0] + pr, u * q[:, 1], q[:, 0]], dim=1)
            Fy = torch.stack([v * q[:, 0], v * q[:, 1] + pr, q[:, 1]], dim=1)
            src = torch.stack([H * self.dh[0], H * self.dh[1], z], dim=1)
            self.vel = [[t[:, 0] / t[:, 2], t[:, 1] / t[:, 2]] for t in own]
        else:
            Fx = torch.stack([u * q[:, 0] + p, u * q[:, 1], q[:, 0], u * rh], dim=1)
            Fy = torch.stack([v * q[:, 0], v * q[:, 1] + p, q[:, 1], v * rh], dim=1)
            if self.env is None:
                src = torch.zeros_like(q)
            else:
                gx, gy = self.env
                cd = 0.0 if case["kind"] == "operators" else 0.01  # the operator's source has no drag
                src = torch.stack([-q[:, 2] * gx - cd * q[:, 0], -q[:, 2] * gy - cd * q[:, 1], z,
                                   -q[:, 0] * gx - q[:, 0] * gy], dim=1)
            if case.get("closure", "off") != "off":
                if first:
                    self.nu = self.viscosity(q)
                gr = [self.nu[:, None, None, None] * t for t in g.gradient_br(q, avg)]
                Fx, Fy = Fx - gr[0], Fy - gr[1]
                bx, by = g.trace(gr[0]), g.trace(gr[1])
                ex, ey = g.neighbour(bx), g.neighbour(by)
                for s in range(4):
                    a, b = (t.unsqueeze(1) for t in g.nh[s])
                    fv = -0.5 * ((bx[s] + ex[s]) * a + (by[s] + ey[s]) * b) * g.ns[s].unsqueeze(1)
                    fv[g.wall(s)] = 0.0
                    fb[s] = fb[s] + fv
        return src - g.divergence(Fx, Fy, fb)

    def steps(self, n, dt):
        q, G = self.q, torch.zeros_like(self.q)
        for _ in range(n):
            for m in range(3):
                G = RK_A[m] * G + self.tendency(q, m == 0)
                q = q + RK_G[m] * (dt if torch.is_tensor(dt) else float(dt)) * G
        self.q = q
        return q

    def entropy(self):
        q, g = self.q, self.g
        if self.model == "lsw":
            e = 0.5 * (self.H * (q[:, 0] ** 2 + q[:, 1] ** 2) + q[:, 2] ** 2)
        elif self.model == "sw":
            e = 0.5 * (q[:, 0] ** 2 + q[:, 1] ** 2) / q[:, 2] + 0.5 * q[:, 2] ** 2 - q[:, 2] * self.top
        else:
            p = self.aux(q)[2]
            e = q[:, 2] * (torch.log(p) - GAMMA * torch.log(q[:, 2])) / (GAMMA - 1)
        return float(g.integral(e))


def _features(q, N):
    """(nEl, 36) closure features and the density's modal decay log10 of a (nEl, 4, P, P) state."""
    P = N + 1
    x, w = np.polynomial.legendre.leggauss(P)
    T = torch.as_tensor((np.polynomial.legendre.legvander(x, N) * np.sqrt(np.arange(P) + 0.5) * w[:, None]).T,
                        device=q.device)
    c = torch.einsum("ki,evji,lj->evkl", T, q[:, 2:4], T) ** 2  # energies [density, total energy]
    tot = c.sum(dim=(2, 3))
    mx = torch.maximum(torch.arange(P)[:, None], torch.arange(P)[None, :]).to(q.device)
    out = []
    for v in range(2):
        for grp in range(3):
            for m in range(N - 5, N + 1):
                e = (c[:, v] * (mx == m)).sum(dim=(1, 2)) if grp == 0 else \
                    c[:, v, m].sum(dim=1) if grp == 1 else c[:, v, :, m].sum(dim=1)
                out.append((torch.log10((e / tot[:, v]).clamp(min=1e-16)) + 8.0) / 8.0)
    top = (c[:, 0] * (mx == N)).sum(dim=(1, 2))
    s = torch.where(top > 0, torch.log10(top / tot[:, 0]), torch.full_like(top, -99.0))
    return torch.stack(out, dim=1), s


def _activation(s, s0):
    ramp = 0.5 * (1.0 + torch.sin(math.pi * (s - s0) / 2.0))
    return torch.where(s < s0 - 1.0, torch.zeros_like(s), torch.where(s > s0 + 1.0, torch.ones_like(s), ramp))


def _mlp_out(params, feat):
    """Clamped output of the network with weights rounded to bfloat16, summed in 64 bits."""
    p = torch.as_tensor(np.asarray(params, dtype=np.float32), device=feat.device)
    r = lambda t: t.to(torch.bfloat16).double()  # noqa: E731
    W1, b1, W2, b2, w3, b3 = torch.split(p, [1152, 32, 1024, 32, 32, 1])
    h = torch.relu(feat @ r(W1).reshape(32, 36).T + b1.double())
    h = torch.relu(h @ r(W2).reshape(32, 32).T + b2.double())
    return (h @ r(w3) + b3.double()).clamp(0.0, 1.0)


def _exact_fields(case, seed):
    g = _Grid(case["N"], case["nx"], case["ny"], False, 0.02)
    r = _rng(seed, 1)
    f = torch.stack([1.0 + _wave(g.X, g.Y, r) for _ in range(case["nVar"])], dim=1)
    bn = torch.as_tensor(0.01 * r.standard_normal((1, 4, case["nVar"], case["N"] + 1)), device=f.device)
    own = g.trace(f)
    gx, gy = g.gradient_br(f, [0.5 * (a + b) for a, b in zip(own, g.neighbour(own))])
    bx, by = g.trace(gx), g.trace(gy)
    n = f.shape[0]
    B = torch.as_tensor(np.stack([g.basis(t) for t in np.linspace(-1.0, 1.0, case["M"] + 1)]), device=f.device)
    return {"gradient boundary": torch.stack([torch.stack(bx, 1), torch.stack(by, 1)], dim=-1),
            "gradient ext": torch.stack([torch.stack(g.neighbour(bx), 1), torch.stack(g.neighbour(by), 1)], dim=-1),
            "divergence": g.divergence(gx, gy, [bn[:, s].expand(n, -1, -1) for s in range(4)]),
            "plot": torch.einsum("ai,evji,bj->evba", B, f, B), "integral": float(g.integral(f[:, 0]))}


def _exact_ensemble(case, seed):
    out = {}
    inst = _members(case, seed)
    for N in sorted({i.N for i in inst}):
        sols = []
        for i in (m for m in inst if m.N == N):
            c = {"kind": "solve", "model": "sw", "N": N, "nx": i.nx, "ny": i.ny, "walls": True, "perturb": 0.0,
                 "sources": False}
            p = _Plain(c, 0)
            g = p.g
            p.top = E.topography(i, g.X, g.Y, xp=torch)
            p.dh = g.gradient_sf(p.top)
            z = torch.zeros_like(g.X)
            p.q = torch.stack([z, z, E.thickness(i, g.X, g.Y, xp=torch)], dim=1)
            p.vel = [[s[:, 0] / s[:, 2], s[:, 1] / s[:, 2]] for s in g.trace(p.q)]
            arc = min(1.0 / i.nx, 1.0 / i.ny) / N ** 2
            sols.append(p.steps(case["steps"], 0.5 * arc / math.sqrt(float(p.q[:, 2].max()))))
        out["N%d" % N] = torch.cat(sols)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "tendency", "operators"):
        c = dict(case)
        if kind == "operators":
            c.update(walls=True, perturb=0.02, model="cig", sources=True)
        p = _Plain(c, seed)
        if kind == "tendency":
            return {"dSdt": p.tendency(p.q)}
        if kind == "operators":
            d = p.tendency(p.q)
            return {"dSdt": d, "q": p.q + RK_G[0] * _dt(case) * d}
        out = {"solution": p.steps(case["steps"], _dt(case))}
        if case["entropy"]:
            out["entropy"] = p.entropy()
        return out
    if kind == "fields":
        return _exact_fields(case, seed)
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    # the features and activations; the trained weights have no value of their own (each step's rounding of the
    # weights to bfloat16 amplifies any difference)
    feat, s = _features(_modal_states(case["N"], case["n"], seed, _device()), case["N"])
    return {"activation": _activation(s, -4.0 * math.log10(case["N"])), "features": feat, "parameters": None,
            "loss": None, "output": None}

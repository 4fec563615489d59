"""The kernels' branches at the sizes where they can go wrong: tiles of odd
degrees, the launch that keeps a mesh on chip, the plane-wise operators, the
reductions and the closure network's tiles."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests import cases as C

pytestmark = pytest.mark.gpu
TOL = 1e-12  # relative per field, as in test_gpu_engine


def _pair(model, kw, N, form, seed=3):
    """The same mesh, fields and state in the oracle and in the engine."""
    import self_b200 as S
    om, pm = C.oracle_mesh(kw), C.product_mesh(kw)
    ref = O.Model(C.MODELS[model], N, om)
    x = O.Geometry(N, om).x
    cls = {"LSW": S.LinearShallowWater, "SW": S.ShallowWater, "CIG": S.CompressibleIdealGas2D}[model]
    mod = cls(pm, S.SEMQuad(S.Lagrange(N, S.GAUSS, N, S.UNIFORM), pm), form=form)
    aux = C.aux_fields(model, x, seed)
    for k, v in aux.items():
        ref.set(k, v)
    if model == "LSW":
        mod.SetBathymetry(aux["H"])
        mod.SetCoriolis(aux["fCori"])
    elif model == "SW":
        mod.SetTopography(aux["topography"])
    else:
        mod.SetGravity(aux["gravityPotential"])
        mod.SetDrag(aux["drag"])
    q = C.initial_state(model, x, seed)
    ref.set("solution", q)
    mod.SetSolution(q)
    return ref, mod, q


def _check(got, ref, form):
    import self_b200 as S
    if form == S.FP64_REF:
        np.testing.assert_array_equal(got, ref)
    else:
        for v in range(ref.shape[2]):
            assert C.rel_err(got[:, :, v], ref[:, :, v]) < TOL


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("model", ["LSW", "SW", "CIG"])
@pytest.mark.parametrize("N", [2, 4, 6])
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 3), (13, 7)])  # odd counts: the last tile is short by any remainder
def test_odd_node_counts_run_the_persistent_kernel(model, N, nx, ny, form):
    """Tendency (reference roundings: bit for bit) and RK3 steps of the persistent kernel at an odd number of nodes,
    where a short last tile leaves copies that are not a multiple of 16 bytes."""
    import self_b200 as S
    kw = dict(nx=nx, ny=ny, bcid=O.BC_NONORMALFLOW, amp=0.03 if nx > 1 else 0.0)
    ref, mod, q = _pair(model, kw, N, form)
    S.check(S.lib().selfgpu_model2d_set_launch(mod._h, 1, 0))
    d = S.to_host(mod.CalculateTendency()).reshape(q.shape, order="F")
    if form == S.FP64_REF:
        np.testing.assert_array_equal(d, ref.tendency())
    mod.SetSolution(q)
    l0 = S.lib().selfgpu_model2d_persistent_launch_count(mod._h)
    mod.ForwardStep(5, 1e-3)
    mod.Sync()
    assert S.lib().selfgpu_model2d_persistent_launch_count(mod._h) - l0 == 15
    ref.rk3(5, 1e-3)
    _check(S.to_host(mod.solution).reshape(q.shape, order="F"), ref.get("solution", q.shape), form)


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("model", ["LSW", "SW", "CIG"])
@pytest.mark.parametrize("N", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("kind", ["single", "torus", "flipped", "ring", "radiation"])
def test_resident_launch_matches_the_oracle(model, N, kind, form):
    """An rk3 call of a small mesh is one launch; over calls of several lengths (odd and even stage counts, stale and
    cached traces) it equals the oracle."""
    import self_b200 as S
    if kind == "radiation" and model == "CIG":
        pytest.skip("zero exterior density")
    ref, mod, q = _pair(model, C.mesh_kwargs(kind), N, form)
    dt = 2e-4
    for n in (1, 2, 3):
        l0 = mod.LaunchCount()
        mod.ForwardStep(n, dt)
        assert mod.LaunchCount() - l0 == 1
        ref.rk3(n, dt)
    mod.Sync()
    _check(S.to_host(mod.solution).reshape(q.shape, order="F"), ref.get("solution", q.shape), form)


@pytest.mark.parametrize("form_name", ["FP64", "FP64_REF", "FP32_BULK"])
@pytest.mark.parametrize("model,N,nx", [("CIG", 7, 33), ("CIG", 7, 52), ("SW", 7, 52), ("LSW", 5, 61), ("SW", 3, 70),
                                        ("CIG", 4, 60), ("SW", 6, 45)])
def test_resident_launch_equals_stage_launches(model, N, nx, form_name):
    """One and several tiles per CTA: the solution and the register of the stage launches bit for bit, with a common
    and with per-element time steps, a tendency between the calls."""
    import self_b200 as S
    out = []
    for pinned in (False, True):
        _, mod, q = _pair(model, dict(nx=nx, ny=nx - 2, periodic=(True, False), bcid=O.BC_NONORMALFLOW, amp=0.02), N,
                          getattr(S, form_name))
        if pinned:
            S.check(S.lib().selfgpu_model2d_set_launch(mod._h, 1, 0))
            S.check(S.lib().selfgpu_model2d_set_multistage(mod._h, 0))
        l0 = mod.LaunchCount()
        mod.ForwardStep(2, 1e-5)
        assert pinned or mod.LaunchCount() - l0 == 1
        mod.CalculateTendency()
        mod._set_field("elementDt", 1e-5 * (1.0 + 0.5 * torch.sin(torch.arange(mod.nElem, device="cuda").double())))
        mod.ForwardStep(3, 0.0)
        mod.Sync()
        out.append((mod.solution.clone(), mod.workSol.clone(), mod.CalculateTendency().clone()))
    assert torch.isfinite(out[0][0]).all()
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_resident_exchange_wait_is_bounded():
    """One CTA publishes no traces: its neighbours' waits run out, sync reports it, and the handle then runs again."""
    import self_b200 as S
    L = S.lib()
    _, mod, q = _pair("CIG", C.mesh_kwargs("periodic"), 7, S.FP64)
    assert L.selfgpu_model2d_set_wait_limit(mod._h, 20_000_000) == 0  # ~10 ms
    assert L.selfgpu_model2d_inject_stall(mod._h, 2) == 0
    mod.ForwardStep(2, 1e-4)
    with pytest.raises(S.SelfGpuError) as ei:
        mod.Sync()
    assert ei.value.code == 6
    assert L.selfgpu_model2d_inject_stall(mod._h, 0) == 0
    ref, _, _ = _pair("CIG", C.mesh_kwargs("periodic"), 7, S.FP64)
    mod.SetSolution(q)
    mod.ForwardStep(3, 1e-4)
    mod.Sync()
    ref.rk3(3, 1e-4)
    _check(S.to_host(mod.solution).reshape(q.shape, order="F"), ref.get("solution", q.shape), S.FP64)


def test_one_sided_neighbours_keep_stage_launches():
    """A mesh whose sideInfo names a neighbour that does not name it back: no exchange of published traces."""
    import self_b200 as S
    m = S.Mesh2D(4, 3, periodic=(True, True))
    si = m.sideInfo.copy(order="F")
    si[2, 1, 0], si[3, 1, 0] = 7, 41  # east side of element 1: the west side of element 7 (not its true neighbour)
    mesh = S.Mesh2D.from_arrays(m.nodeCoords, si)
    mod = S.CompressibleIdealGas2D(mesh, S.SEMQuad(S.Lagrange(5, S.GAUSS, 5, S.UNIFORM), mesh))
    q = torch.ones_like(mod.solution)
    q[:, 3] = 3.0
    mod.SetSolution(q)
    l0 = mod.LaunchCount()
    mod.ForwardStep(2, 1e-5)
    mod.Sync()
    assert mod.LaunchCount() - l0 == 1 + 6


@pytest.mark.parametrize("N", [2, 3, 6, 7, 8, 10])
@pytest.mark.parametrize("nVar,nEl", [(1, 1), (3, 5), (2, 131)])
def test_plane_operators_match_the_oracle(N, nVar, nEl):
    """The operators that take several planes per block, at plane counts that leave the last block short, and the
    degrees beyond the compiled ones: bit for bit the oracle's."""
    import self_b200 as S
    P, w = N + 1, S.lib()
    Lo = O.Lagrange(N, O.GAUSS, 5, O.UNIFORM)
    om = O.Mesh(nEl, 1, periodic=(True, False), bcid=O.BC_NONORMALFLOW)
    g = O.Geometry(N, om)
    r = np.random.default_rng(N + nEl)
    f = np.asfortranarray(r.standard_normal((P, P, nVar, nEl)))
    v = np.asfortranarray(r.standard_normal((2, P, P, nVar, nEl)))
    avg = np.asfortranarray(r.standard_normal((P, nVar, 4, nEl)))
    p = lambda t: S._lib.pp(t.data_ptr())  # noqa: E731
    dev = {k: S.to_device(a) for k, a in dict(f=f, v=v, avg=avg, dsdx=g.dsdx, J=g.J, nHat=g.nHat, nScale=g.nScale,
                                               **{m: getattr(Lo, m) for m in ("iMatrix", "dMatrix", "dgMatrix",
                                                                              "bMatrix", "qWeights")}).items()}
    a = {k: p(t) for k, t in dev.items()}

    def run(call, shape, *args):
        out = S.to_device(np.zeros(shape, order="F"))
        call(*[p(out) if x is None else x for x in args])
        torch.cuda.synchronize()
        return S.to_host(out).reshape(shape, order="F")

    n = (N, nVar, nEl)
    eq = np.testing.assert_array_equal
    eq(run(w.ScalarGridInterp_2D_gpu_wrapper, (6, 6, nVar, nEl), a["iMatrix"], a["f"], None, N, 5, nVar, nEl),
       O.scalar_grid_interp(Lo, f))
    eq(run(w.VectorGridInterp_2D_gpu_wrapper, (2, 6, 6, nVar, nEl), a["iMatrix"], a["v"], None, N, 5, nVar, nEl),
       O.vector_grid_interp(Lo, v))
    eq(run(w.ScalarBoundaryInterp_2D_gpu_wrapper, (P, nVar, 4, nEl), a["bMatrix"], a["f"], None, *n),
       O.scalar_boundary_interp(Lo, f))
    eq(run(w.VectorBoundaryInterp_2D_gpu_wrapper, (2, P, nVar, 4, nEl), a["bMatrix"], a["v"], None, *n),
       O.vector_boundary_interp(Lo, v))
    eq(run(w.VectorGradient_2D_gpu_wrapper, (2, 2, P, P, nVar, nEl), a["dMatrix"], a["v"], None, *n),
       O.vector_gradient(Lo, v))
    eq(run(w.VectorDGDivergence_2D_gpu_wrapper, (P, P, nVar, nEl), a["dgMatrix"], a["bMatrix"], a["qWeights"], a["v"],
           a["avg"], None, *n), O.vector_dg_divergence(Lo, v, avg))
    eq(run(w.GradientSF_MappedScalar2D_gpu_wrapper, (2, P, P, nVar, nEl), a["f"], a["dsdx"], a["J"], None,
           a["dMatrix"], *n), O.gradient_sf(Lo, f, g.dsdx, g.J))
    eq(run(w.GradientBR_MappedScalar2D_gpu_wrapper, (2, P, P, nVar, nEl), a["f"], a["avg"], a["dsdx"], a["J"],
           a["nHat"], a["nScale"], None, a["dgMatrix"], a["bMatrix"], a["qWeights"], *n),
       O.gradient_br(Lo, f, avg, g.dsdx, g.J, g.nHat, g.nScale))


@pytest.mark.parametrize("N,nx,ny", [(2, 1, 1), (3, 17, 5), (7, 40, 37)])  # one block; several; more than one sweep
def test_integral_and_entropy_sums(N, nx, ny):
    """The reductions against their defining sums in long double; 1e-13 relative to the sum of magnitudes (a pairwise
    sum of n <= 1e5 terms rounds to far below n eps)."""
    import self_b200 as S
    ref, mod, q = _pair("CIG", dict(nx=nx, ny=ny, bcid=O.BC_NONORMALFLOW, amp=0.0), N, S.FP64)
    wJ = S.to_host(mod._wJ()).astype(np.longdouble)  # (P, P, nEl)
    f = S.MappedScalar2D(mod.interp, 4, mod.nElem)
    f.interior.copy_(mod.solution)
    for v in range(4):
        terms = q[:, :, v].astype(np.longdouble) * wJ
        assert abs(f.Integral(mod.geometry, v + 1) - float(terms.sum())) <= 1e-13 * float(np.abs(terms).sum())
    ru, rv, r, e = (q[:, :, k].astype(np.longdouble) for k in range(4))
    p = 0.4 * (e - 0.5 * (ru * ru + rv * rv) / r)
    terms = r * (np.log(p) - 1.4 * np.log(r)) / 0.4 * wJ
    for _ in range(2):  # the scratch is left as it was found
        assert abs(mod.CalculateEntropy() - float(terms.sum())) <= 1e-13 * float(np.abs(terms).sum())


def _mix64(x):
    x = (x + np.uint64(0x9E3779B97F4A7C15)).astype(np.uint64)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


@pytest.mark.parametrize("n,batch", [(40, 1), (100, 31), (100, 33), (3000, 9473)])  # tiles of 32, 296 blocks
def test_training_steps_match_float64(n, batch):
    """Two epochs of Adam against the same steps in float64: the losses to 1e-4 (float32 sums; 1e-2 over 80 steps, in
    which a weight near a bfloat16 midpoint may round the other way for the forward pass), and a second run bit for
    bit the first."""
    from self_b200 import closure as CL
    r = np.random.default_rng(n)
    feat = r.uniform(0, 1, (n, 36)).astype(np.float32)
    y = np.clip(2.0 * feat[:, 5] - 0.5, 0, 1).astype(np.float32)
    F, Y = torch.from_numpy(feat).cuda(), torch.from_numpy(y).cuda()
    m = CL.ClosureMLP(seed=2)
    p0 = m.params.copy()
    loss = m.train(F, Y, epochs=2, batch=batch, lr=1e-3, seed=9)
    m2 = CL.ClosureMLP(params=p0.copy())
    loss2 = m2.train(F, Y, epochs=2, batch=batch, lr=1e-3, seed=9)
    np.testing.assert_array_equal(m.params, m2.params)
    np.testing.assert_array_equal(loss, loss2)
    p = p0.astype(np.float64)
    m1, v1 = np.zeros_like(p), np.zeros_like(p)
    cuts = np.cumsum([1152, 32, 1024, 32, 32])
    steps, ref, t = -(-n // batch), [], 0
    with np.errstate(over="ignore"):
        for _ in range(2):
            tot = 0.0
            for _ in range(steps):
                k = np.uint64(t) * np.uint64(0x100000001) + np.arange(batch, dtype=np.uint64)
                idx = (_mix64(np.uint64(9) ^ _mix64(k)) % np.uint64(n)).astype(np.int64)
                W1, b1, W2, b2, w3, b3 = np.split(p, cuts)
                rnd = lambda a: O.bf16_round(a.astype(np.float32)).astype(np.float64)  # noqa: E731
                W1, W2, w3 = rnd(W1).reshape(32, 36), rnd(W2).reshape(32, 32), rnd(w3)
                x, lab = feat[idx].astype(np.float64), y[idx].astype(np.float64)
                h1 = np.maximum(x @ W1.T + b1, 0)
                h2 = np.maximum(h1 @ W2.T + b2, 0)
                z = h2 @ w3 + b3
                a = np.clip(z, 0, 1)
                d = np.where(((z < 0) & (lab > 0)) | ((z > 1) & (lab < 1)), z - lab, a - lab)
                tot += ((a - lab) ** 2).sum()
                gz = 2 * d / batch
                d2 = gz[:, None] * w3 * (h2 > 0)
                d1 = (d2 @ W2) * (h1 > 0)
                g = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ gz,
                                    [gz.sum()]])
                t += 1
                m1, v1 = 0.9 * m1 + 0.1 * g, 0.999 * v1 + 0.001 * g * g
                p = p - 1e-3 * (m1 / (1 - 0.9 ** t)) / (np.sqrt(v1 / (1 - 0.999 ** t)) + 1e-8)
            ref.append(tot / (steps * batch))
    np.testing.assert_allclose(loss, ref, rtol=1e-2 if steps > 4 else 1e-4)


@pytest.mark.parametrize("n", [1, 7, 1185, 30001])  # fewer rows than a block's; one row more than a sweep; several
@pytest.mark.parametrize("nan", [False, True])
def test_feature_range_of_a_training_set(n, nan):
    from self_b200 import closure as CL
    f = np.random.default_rng(n).standard_normal((n, 36)).astype(np.float32)
    if nan:
        f[n // 2, 5] = np.nan
    m = CL.ClosureMLP(seed=0)
    m.train(torch.from_numpy(f).cuda(), torch.zeros(n, device="cuda"), epochs=0, batch=8)
    np.testing.assert_array_equal(m.fmin, f.min(axis=0))
    np.testing.assert_array_equal(m.fmax, f.max(axis=0))


@pytest.mark.parametrize("n", [1, 31, 33, 37921])  # a short tile; more tiles than blocks
def test_inference_tiles(n):
    """The clamped output against the restatement, to 1e-5 (float32 sums of 36 and 32 products of order one)."""
    from self_b200 import closure as CL
    m = CL.ClosureMLP(seed=5)
    f = np.random.default_rng(n).uniform(-1, 1, (n, 36)).astype(np.float32)
    got = m.infer(torch.from_numpy(f).cuda()).cpu().numpy()
    assert np.abs(got - O.mlp_forward(f.T, *m.unpack())).max() < 1e-5


@pytest.mark.parametrize("N", [2, 4, 6])
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (131, 41)])  # less than a warp's elements; a short one; several blocks
def test_closure_lane_groups(N, nx, ny):
    """Eight lanes per element: groups without an element, and fewer node rows than lanes, against the oracle."""
    import self_b200 as S
    kw = dict(nx=nx, ny=ny, periodic=(False, False), bcid=O.BC_NONORMALFLOW, amp=0.02 if nx > 1 else 0.0)
    ref, mod, _ = _pair("CIG", kw, N, S.FP64)
    q = C.shock_state(O.Geometry(N, C.oracle_mesh(kw)).x, 1)
    ref.set("solution", q)
    mod.SetSolution(q)
    ref.set_closure(1, c=1.0)
    mod.SetClosure(S.CLOSURE_INDICATOR, c=1.0)
    t = ref.tendency()
    got = S.to_host(mod.CalculateTendency()).reshape(t.shape, order="F")
    nu = ref.get("avNu")
    assert np.abs(mod.ClosureState()[0].cpu().numpy() - nu).max() <= 1e-13 * nu.max()
    _check(got, t, S.FP64)


def test_gas_entropy_of_a_state_whose_squares_overflow():
    """The pressure is formed from rho u times u, as the reference forms it: momenta above 1.4e154, whose squares
    overflow, in a fluid as dense."""
    import self_b200 as S
    mesh = S.Mesh2D(3, 2, periodic=(True, True))
    m = S.CompressibleIdealGas2D(mesh, S.SEMQuad(S.Lagrange(3, S.GAUSS, 3, S.UNIFORM), mesh))
    q = torch.empty_like(m.solution)
    q[:, 0], q[:, 1], q[:, 2], q[:, 3] = 3e154, -2e154, 2e154, 1e155
    m.SetSolution(q)
    r, e = np.longdouble(2e154), np.longdouble(1e155)
    p = 0.4 * (e - 0.5 * (np.longdouble(3e154) * 1.5 + np.longdouble(2e154)))
    ref = float(r * (np.log(p) - 1.4 * np.log(r)) / 0.4)  # of a unit square
    assert abs(m.CalculateEntropy() - ref) <= 1e-13 * abs(ref)

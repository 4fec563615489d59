"""Degree 1 (two nodes per direction), with operators from its Gauss nodes
+-1/sqrt(3): the set-up routines follow the reference's, whose quadrature is
degenerate there, so a caller brings its own matrices and geometry."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
A = 1.0 / np.sqrt(3.0)


def interp():
    import self_b200 as S
    L = S.Lagrange(1, S.GAUSS, 1, S.UNIFORM)
    L.controlPoints[:] = -A, A
    L.qWeights[:] = 1.0
    L.dMatrix[:] = [[-0.5 / A] * 2, [0.5 / A] * 2]  # l_ii'(x_i) at (ii, i)
    L.dgMatrix[:] = -L.dMatrix.T
    L.bMatrix[:] = [[(1 + A) / (2 * A), (A - 1) / (2 * A)], [(A - 1) / (2 * A), (1 + A) / (2 * A)]]
    return L


def geometry(mesh, nx, ny):
    """Rectangles of 1/nx by 1/ny."""
    import self_b200 as S
    geo = S.SEMQuad(interp(), mesh)
    hx, hy = 1.0 / nx, 1.0 / ny
    e = torch.arange(nx * ny, device="cuda")
    x = torch.tensor([-A, A], device="cuda", dtype=torch.float64)
    geo.x[..., 0] = ((e % nx).double() * hx)[:, None, None, None] + 0.5 * hx * (1 + x)[None, None, None, :]
    geo.x[..., 1] = ((e // nx).double() * hy)[:, None, None, None] + 0.5 * hy * (1 + x)[None, None, :, None]
    geo.dsdx[:] = torch.tensor([[hy / 2, 0.0], [0.0, hx / 2]], device="cuda", dtype=torch.float64)
    geo.J[:] = hx * hy / 4
    n = torch.tensor([[0.0, -1.0], [1.0, 0.0], [0.0, 1.0], [-1.0, 0.0]], device="cuda", dtype=torch.float64)
    geo.nHat[:] = n[None, :, None, None, :]
    w = torch.tensor([hx / 2, hy / 2, hx / 2, hy / 2], device="cuda", dtype=torch.float64)
    geo.nScale[:] = w[None, :, None, None]
    return geo


def model(name, nx, ny, form):
    import self_b200 as S
    mesh = S.Mesh2D(nx, ny, periodic=(True, False), bcid=S.BC_NONORMALFLOW)
    geo = geometry(mesh, nx, ny)
    m = {"LSW": S.LinearShallowWater, "SW": S.ShallowWater, "CIG": S.CompressibleIdealGas2D}[name](mesh, geo, form=form)
    if name == "LSW":
        ones = torch.ones((nx * ny, 1, 2, 2), device="cuda", dtype=torch.float64)
        m._set_field("H", ones)
        m._set_field("H.boundary", torch.ones((nx * ny, 4, 1, 2), device="cuda", dtype=torch.float64))
    return m, geo


@pytest.mark.parametrize("nx,ny", [(5, 3), (60, 41)])
@pytest.mark.parametrize("form_name", ["FP64", "FP64_REF", "FP32_BULK"])
def test_a_linear_surface_has_its_exact_gradient(form_name, nx, ny):
    """eta = x, at rest, H = g = 1: (du/dt, dv/dt, deta/dt) = (-1, 0, 0) away from the seam of the periodic direction
    (the two columns of elements whose traces meet the jump) and, for v, from the walls."""
    import self_b200 as S
    m, geo = model("LSW", nx, ny, getattr(S, form_name))
    q = torch.zeros_like(m.solution)
    q[:, 2] = geo.x[:, 0, :, :, 0]
    m.SetSolution(q)
    d = m.CalculateTendency().reshape(ny, nx, 3, 2, 2)
    # a difference of fluxes of order one, some fifty roundings, over half an element's width
    tol = 100.0 * (2.0 ** -24 if form_name == "FP32_BULK" else 2.0 ** -53) * max(nx, ny)
    inner = d[1:-1, 1:-1]
    assert (inner[:, :, 0] + 1.0).abs().max() < tol and inner[:, :, 1:].abs().max() < tol


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 3), (70, 33), (131, 41)])  # one and several tiles per CTA
@pytest.mark.parametrize("form_name", ["FP64", "FP64_REF", "FP32_BULK"])
@pytest.mark.parametrize("name", ["LSW", "SW", "CIG"])
def test_the_three_kernels_agree(name, form_name, nx, ny):
    """Steps on chip, as launches of the persistent kernel and of the per-element kernel: the first two bit for bit,
    the third bit for bit with the reference's roundings and to the rounding of the form (1e-12, 1e-5) otherwise."""
    import self_b200 as S
    out = []
    for kernel in ("chip", 1, 0):
        m, geo = model(name, nx, ny, getattr(S, form_name))
        X, Y = geo.x[:, 0, :, :, 0], geo.x[:, 0, :, :, 1]
        q = torch.zeros_like(m.solution)
        q[:, 0] = 0.1 * torch.sin(2 * np.pi * Y)
        q[:, 2] = 1.0 + 0.05 * torch.sin(2 * np.pi * X) * torch.cos(2 * np.pi * Y)
        if name == "CIG":
            q[:, 3] = 2.5 + 0.1 * torch.cos(2 * np.pi * X)
        if kernel != "chip":
            S.check(S.lib().selfgpu_model2d_set_launch(m._h, kernel, 0))
        m.SetSolution(q)
        l0 = m.LaunchCount()
        m.ForwardStep(2, 1e-3 / max(nx, ny))
        assert m.LaunchCount() - l0 == (1 if kernel == "chip" else 7)
        m.ForwardStep(3, 1e-3 / max(nx, ny))
        m.Sync()
        out.append((m.solution.clone(), m.CalculateTendency().clone()))
    assert torch.isfinite(out[0][1]).all()
    tol = 1e-5 if form_name == "FP32_BULK" else 1e-12
    for chip, persistent, element in zip(*out):
        assert torch.equal(chip, persistent)
        if form_name == "FP64_REF":
            assert torch.equal(chip, element)
    for v in range(out[0][0].shape[1]):  # the states
        a, b = out[0][0][:, v], out[2][0][:, v]
        assert (a - b).abs().max() <= tol * max(float(b.abs().max()), 0.1)


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (131, 41)])
def test_the_indicator_closure(nx, ny):
    """Element viscosity (two lanes per element) and the features' activation against their definition."""
    import self_b200 as S
    from self_b200 import closure as CL
    m, geo = model("CIG", nx, ny, S.FP64)
    r = np.random.default_rng(nx)
    q = np.zeros((nx * ny, 4, 2, 2))
    q[:, 2] = r.uniform(0.5, 1.5, (nx * ny, 1, 1)) + r.uniform(-0.3, 0.3, (nx * ny, 2, 2))
    q[:, 0] = 0.2 * q[:, 2]
    q[:, 3] = 2.5
    m.SetSolution(torch.from_numpy(q).cuda())
    m.SetClosure(S.CLOSURE_INDICATOR, c=0.5, s0=-1.0, kappa=1.0)
    assert torch.isfinite(m.CalculateTendency()).all()
    nu, act = (x.cpu().numpy() for x in m.ClosureState()[:2])
    T = np.array([[np.sqrt(0.5), np.sqrt(0.5)], [-np.sqrt(1.5) * A, np.sqrt(1.5) * A]])  # w_i Lt_k(x_i)
    c = np.einsum("li,eij,kj->elk", T, q[:, 2], T) ** 2
    s = np.log10((c[:, 0, 1] + c[:, 1, 0] + c[:, 1, 1]) / c.sum((1, 2)))
    a = np.where(s < -2.0, 0.0, np.where(s > 0.0, 1.0, 0.5 * (1 + np.sin(np.pi * (s + 1.0) / 2))))
    p = 0.4 * (q[:, 3] - 0.5 * q[:, 0] ** 2 / q[:, 2])
    lam = (np.abs(q[:, 0] / q[:, 2]) + np.sqrt(1.4 * p / q[:, 2])).max((1, 2))
    ref = a * 0.5 * np.sqrt(1.0 / (nx * ny)) * lam
    assert 0 < np.count_nonzero(ref)
    assert np.abs(nu - ref).max() < 1e-12 * ref.max()
    assert np.abs(act - a).max() < 1e-6
    got, _ = CL.features(torch.from_numpy(q).cuda(), m.interp, s0=-1.0)
    assert np.abs(got.cpu().numpy() - a).max() < 1e-6

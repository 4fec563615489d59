"""How the RK3 steps of a call reach the device: refused and bounded
cooperative launches, captured calls, tuned launches."""
import pytest
import torch

from tests import launch_shim

pytestmark = pytest.mark.gpu


def model(name, nx, N, form, stream=None, ny=None):
    """A periodic mesh with perturbed nodes and a smooth state."""
    import self_b200 as S
    mesh = S.Mesh2D(nx, ny or nx, periodic=(True, True), perturbation=0.02)
    geo = S.SEMQuad(S.Lagrange(N, S.GAUSS, N, S.UNIFORM), mesh)
    m = {"LSW": S.LinearShallowWater, "SW": S.ShallowWater, "CIG": S.CompressibleIdealGas2D}[name](
        mesh, geo, form=form, stream=stream)
    q = torch.zeros_like(m.solution)
    q[:, 0], q[:, 2] = 0.1, 1.0 + 0.05 * torch.sin(6.28 * geo.x[:, 0, :, :, 0])
    if name == "CIG":
        q[:, 3] = 2.5
    m.SetSolution(q)
    return m


def refused(nx):
    """Two steps where the runtime refuses cooperative launches, and as pinned stage launches."""
    import self_b200 as S
    a, b = (model("CIG", nx, 7, S.FP64) for _ in range(2))
    l0 = a.LaunchCount()
    a.ForwardStep(2, 1e-5)
    a.Sync()
    assert a.LaunchCount() - l0 == 1 + 6, a.LaunchCount() - l0  # the trace prologue, then a launch per stage
    S.check(S.lib().selfgpu_model2d_set_launch(b._h, 1, 0))
    S.check(S.lib().selfgpu_model2d_set_multistage(b._h, 0))
    b.ForwardStep(2, 1e-5)
    b.Sync()
    assert torch.isfinite(a.solution).all() and torch.equal(a.solution, b.solution)


@pytest.mark.parametrize("nx", [9, 80])  # where the on-chip and where the multi-stage launch would run
def test_a_refused_cooperative_launch_runs_stage_launches(nx, tmp_path):
    noted = launch_shim.run(tmp_path, f"from tests.test_gpu_launches import refused; refused({nx})", refuse=True)
    assert any(cooperative for _, cooperative in noted)


@pytest.mark.parametrize("name", ["LSW", "SW"])
def test_a_long_call_is_several_bounded_launches(name):
    """An on-chip launch holds its SMs: 2 001 steps are three launches, with the state of the stage launches."""
    import self_b200 as S
    out = []
    for pinned in (False, True):
        m = model(name, 5, 3, S.FP64)
        if pinned:
            S.check(S.lib().selfgpu_model2d_set_launch(m._h, 1, 0))
        l0 = m.LaunchCount()
        m.ForwardStep(2001, 1e-5)
        m.Sync()
        assert pinned or m.LaunchCount() - l0 == 3
        out.append((m.solution.clone(), m.workSol.clone()))
    assert torch.isfinite(out[0][0]).all()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("name,nx,N", [("LSW", 8, 7), ("SW", 24, 7), ("SW", 90, 4), ("CIG", 50, 7), ("CIG", 9, 2)])
def test_a_captured_call_replays(name, nx, N, n):
    """An on-chip call captured into a CUDA graph, with an odd or an even number of steps, and replayed: the steps of
    as many calls, bit for bit (one and several tiles per CTA)."""
    import self_b200 as S
    st = torch.cuda.Stream()
    a, b = (model(name, nx, N, S.FP64, stream=s) for s in (st.cuda_stream, None))
    torch.cuda.synchronize()
    for m in (a, b):
        m.ForwardStep(1, 1e-5)
        m.Sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        a.ForwardStep(n, 1e-5)
    for _ in range(4):
        graph.replay()
    torch.cuda.synchronize()
    a.ForwardStep(2, 1e-5)
    a.Sync()
    for _ in range(4):
        b.ForwardStep(n, 1e-5)
    b.ForwardStep(2, 1e-5)
    b.Sync()
    assert torch.isfinite(a.solution).all()
    assert torch.equal(a.solution, b.solution) and torch.equal(a.workSol, b.workSol)

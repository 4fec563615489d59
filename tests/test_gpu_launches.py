"""How the RK3 steps of a call reach the device: refused and bounded
cooperative launches, captured calls, tuned launches."""
import ctypes
from collections import Counter

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
    assert any(cooperative for stretch in noted for _, cooperative in stretch)


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


def tuned(name, nx, ny, N, form_name):
    """A step of stage launches as configured by default, the autotuner, and then steps of a new solution."""
    import self_b200 as S
    L = S.lib()
    m = model(name, nx, N, getattr(S, form_name), ny=ny)
    S.check(L.selfgpu_model2d_set_multistep(m._h, 0))
    launch_shim.mark()
    m.ForwardStep(1, 1e-5)
    launch_shim.mark()
    p, c, us = ctypes.c_int(), ctypes.c_int(), ctypes.c_float()
    S.check(L.selfgpu_model2d_autotune(m._h, ctypes.byref(p), ctypes.byref(c), ctypes.byref(us)))
    launch_shim.mark()
    m.ForwardStep(1, 1e-5)
    m.Sync()
    assert (c.value > 0) == bool(p.value) and us.value > 0


@pytest.mark.parametrize("name,nx,ny,N,form_name,threads", [
    ("SW", 9, 7, 4, "FP32_BULK", 64),  # an odd number of values, twelve groups
    ("LSW", 7, 5, 6, "FP64", 128), ("CIG", 9, 7, 2, "FP64", 96), ("SW", 8, 8, 7, "FP32_BULK", 64),
    ("CIG", 6, 6, 3, "FP64", 32)])
def test_the_autotuner_times_every_group_count_once(name, nx, ny, N, form_name, threads, tmp_path):
    """Four launches with each number of consumer groups from two to the default, which is the most that fit."""
    noted = launch_shim.run(tmp_path, "from tests.test_gpu_launches import tuned; "
                                      f"tuned({name!r}, {nx}, {ny}, {N}, {form_name!r})")
    _, default, candidates, _ = noted
    assert len(default) == 3 and len(set(default)) == 1
    fit = default[0][0] // threads
    assert fit >= 2 and default[0][0] == fit * threads
    assert Counter(candidates) == {(g * threads, 0): 4 for g in range(2, fit + 1)}


def test_the_autotuner_leaves_the_on_chip_launch():
    """Its choice is for stage launches: rk3 on a mesh that fits on chip stays one launch, with the same state."""
    import self_b200 as S
    L = S.lib()
    a, b = (model("CIG", 9, 5, S.FP64) for _ in range(2))
    p, c, us = ctypes.c_int(), ctypes.c_int(), ctypes.c_float()
    S.check(L.selfgpu_model2d_autotune(a._h, ctypes.byref(p), ctypes.byref(c), ctypes.byref(us)))
    for m in (a, b):
        l0 = m.LaunchCount()
        m.ForwardStep(3, 1e-5)
        m.Sync()
        assert m.LaunchCount() - l0 == 1
    assert torch.equal(a.solution, b.solution)


@pytest.mark.parametrize("name,nx,N,form_name,least", [
    # several tiles per CTA
    ("SW", 38, 7, "FP64_REF", 2), ("CIG", 52, 7, "FP64_REF", 4), ("CIG", 60, 7, "FP64", 2), ("LSW", 60, 5, "FP64", 2),
    ("CIG", 60, 5, "FP32_BULK", 2), ("LSW", 60, 5, "FP32_BULK", 1), ("SW", 90, 4, "FP64", 1),
    ("CIG", 80, 2, "FP32_BULK", 2),
    # one tile; more than the launch gains from
    ("SW", 30, 7, "FP64_REF", 1), ("CIG", 104, 3, "FP64", None), ("SW", 60, 5, "FP64_REF", None),
    ("CIG", 120, 2, "FP32_BULK", None)])
def test_a_call_runs_on_chip_where_that_is_faster(name, nx, N, form_name, least):
    """Calls shorter than the on-chip launch needs to win back its start run stage launches (counted as two steps
    longer where the traces are stale), as do meshes of more tiles than it gains from; the state is the same however
    the steps are divided."""
    import self_b200 as S
    a, b = (model(name, nx, N, getattr(S, form_name)) for _ in range(2))
    S.check(S.lib().selfgpu_model2d_set_launch(b._h, 1, 0))
    stale = True
    for n in (1, 1, 2, 3, 4, 1):
        l0 = a.LaunchCount()
        a.ForwardStep(n, 1e-6)
        on_chip = least is not None and n + 2 * stale >= least
        assert a.LaunchCount() - l0 == (1 if on_chip else 3 * n + stale), (n, stale)
        stale = False
        b.ForwardStep(n, 1e-6)
    a.Sync()
    b.Sync()
    assert torch.isfinite(a.solution).all()
    assert torch.equal(a.solution, b.solution) and torch.equal(a.workSol, b.workSol)


@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("name,nx,N,closure", [
    ("CIG", 100, 3, False), ("SW", 100, 7, False), ("SW", 120, 4, False), ("CIG", 61, 7, False), ("CIG", 20, 5, True)])
def test_captured_stage_launches_replay(name, nx, N, closure, n):
    """Meshes and calls of stage launches (one of them where longer calls run on chip or as one launch), captured after
    a call of another kind: the steps of as many calls, bit for bit."""
    import self_b200 as S
    st = torch.cuda.Stream()
    a, b = (model(name, nx, N, S.FP64, stream=s) for s in (st.cuda_stream, None))
    torch.cuda.synchronize()
    for m in (a, b):
        if closure:
            m.SetClosure(S.CLOSURE_INDICATOR, c=1.0)
        m.ForwardStep(5, 1e-5)
        m.Sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        a.ForwardStep(n, 1e-5)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    a.ForwardStep(4, 1e-5)
    a.Sync()
    for _ in range(3):
        b.ForwardStep(n, 1e-5)
    b.ForwardStep(4, 1e-5)
    b.Sync()
    assert torch.isfinite(a.solution).all()
    assert torch.equal(a.solution, b.solution) and torch.equal(a.workSol, b.workSol)

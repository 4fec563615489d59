"""RK steps as stage launches, which every large mesh runs, on small meshes
that would run the on-chip launch by default."""
import numpy as np
import pytest

from tests import cases as C
from tests.test_gpu_engine import build_oracle, build_pair

pytestmark = pytest.mark.gpu
TOL = 1e-12  # relative per field, as in test_gpu_engine
FORMS = [0, 2]


def stage_launches(mod):
    import self_b200 as S
    S.check(S.lib().selfgpu_model2d_set_launch(mod._h, 1, 0))
    S.check(S.lib().selfgpu_model2d_set_multistage(mod._h, 0))
    return S.lib().selfgpu_model2d_persistent_launch_count(mod._h)


def check(mod_o, mod, form, alt_o):
    """Reference roundings: bit for bit.  Production form: the bound of test_gpu_engine's check_tendency, 1e-12 or 8x
    the oracle's own sensitivity to rounding (alt_o, its contracted build)."""
    import self_b200 as S
    ref = mod_o.get("solution", (mod.N + 1, mod.N + 1, mod.nVar, mod.nElem))
    got = S.to_host(mod.solution).reshape(ref.shape, order="F")
    assert np.isfinite(ref).all()
    if form == S.FP64_REF:
        np.testing.assert_array_equal(got, ref)
    else:
        alt = alt_o.get("solution", ref.shape)
        for v in range(ref.shape[2]):
            bound = max(TOL, 8.0 * C.rel_err(alt[:, :, v], ref[:, :, v]))
            assert C.rel_err(got[:, :, v], ref[:, :, v]) <= bound, (v, bound)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("N", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("model,mesh_kind", [
    (m, k) for m in ("LSW", "SW", "CIG")
    for k in ("periodic", "walls", "flipped", "radiation", "single", "column", "row", "pair", "ring", "torus")
] + [("CIG", "prescribed")])
def test_steps_match_the_oracle(model, mesh_kind, N, form):
    """Every boundary condition, flipped sides and the smallest meshes: twelve steps (graph replays after the first)
    over two calls."""
    import self_b200 as S
    mod_o, mod, _, _ = build_pair(model, mesh_kind, N, seed=3, form=form)
    l0 = stage_launches(mod)
    mod.ForwardStep(5, 1e-3)
    mod.ForwardStep(7, 1e-3)
    mod.Sync()
    assert S.lib().selfgpu_model2d_persistent_launch_count(mod._h) - l0 == 36
    alt_o = build_oracle(model, mesh_kind, N, 3, fast=True)
    for o in (mod_o, alt_o):
        o.rk3(12, 1e-3)
    check(mod_o, mod, form, alt_o)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("model", ["LSW", "SW", "CIG"])
def test_100_steps_match_the_oracle(model, form):
    mesh_kind = "periodic" if model == "CIG" else "walls"
    mod_o, mod, _, _ = build_pair(model, mesh_kind, 7, seed=7, form=form)
    alt_o = build_oracle(model, mesh_kind, 7, 7, fast=True)
    stage_launches(mod)
    for o in (mod_o, alt_o):
        o.rk3(100, 5e-4)
    mod.ForwardStep(40, 5e-4)
    mod.ForwardStep(60, 5e-4)
    mod.Sync()
    check(mod_o, mod, form, alt_o)


@pytest.mark.parametrize("model,N", [("CIG", 7), ("SW", 5), ("LSW", 7), ("SW", 6), ("CIG", 3)])
def test_graph_replays_equal_separate_stages(model, N):
    """Steps replayed from a graph and the same stages issued one by one (the multi-rank entry point), on a mesh with
    several elements per CTA: bit for bit."""
    import self_b200 as S
    L = S.lib()
    n, dt, outs = 4, 2e-4, []
    for graphed in (True, False):
        mesh = S.Mesh2D(24, 20, periodic=(True, True), perturbation=0.05)
        geo = S.SEMQuad(S.Lagrange(N, S.GAUSS, N, S.UNIFORM), mesh)
        mod = {"LSW": S.LinearShallowWater, "SW": S.ShallowWater, "CIG": S.CompressibleIdealGas2D}[model](mesh, geo)
        x = S.to_host(geo.x)
        aux = C.aux_fields(model, x, 9)
        if model == "LSW":
            mod.SetBathymetry(aux["H"])
            mod.SetCoriolis(aux["fCori"])
        elif model == "SW":
            mod.SetTopography(aux["topography"])
        else:
            mod.SetGravity(aux["gravityPotential"])
            mod.SetDrag(aux["drag"])
        mod.SetSolution(C.initial_state(model, x, 9))
        l0 = stage_launches(mod)
        if graphed:
            mod.ForwardStep(n, dt)
            mod.ForwardStep(n, dt)
        else:
            S.check(L.selfgpu_model2d_prologue(mod._h))
            for k in range(6 * n):
                S.check(L.selfgpu_model2d_stage(mod._h, dt, k % 3))
        mod.Sync()
        assert L.selfgpu_model2d_persistent_launch_count(mod._h) - l0 == 6 * n
        outs.append(S.to_host(mod.solution).copy())
    assert np.isfinite(outs[0]).all()
    np.testing.assert_array_equal(outs[0], outs[1])

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

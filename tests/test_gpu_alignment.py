"""Arrays 8 bytes past a 16-byte boundary: the kernels that read x pairs as one access leave them
to kernels that read single values, in every x route (a pass plan, runtime radices, odd lengths,
lengths with a prime factor above 13), for the solve's array and for each predictor field."""
import numpy as np
import pytest

from conftest import rel_l2
from gpu_util import empty_like_dev, from_dev, to_dev

pytestmark = pytest.mark.gpu

SHAPES = [(64, 12, 32), (40, 9, 20), (15, 8, 21), (34, 7, 19), (62, 6, 46)]


def _off(t):
    import torch
    store = torch.empty(t.numel() + 1, dtype=torch.float64, device=t.device)
    view = store[1:].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16 == 8
    return view


@pytest.mark.parametrize("shape", SHAPES)
def test_solve_of_a_misaligned_array(cuda_device, oracle, shape):
    import prj
    import workloads
    nx, ny, nz = shape
    rhs, yu, dx, dz = workloads.poisson_rhs(nx, ny, nz, seed=61)
    b6 = prj.bands(yu, "reference")
    with prj.Plan(nx, nz, ny, dx, dz, b6) as plan:
        t = _off(to_dev(rhs))
        plan.poisson_fp64(t)
        got = from_dev(t)
    want, _ = oracle.poisson(rhs, dx, dz, b6)
    assert rel_l2(got, want) <= 1e-12


@pytest.mark.parametrize("which", [(0,), (1,), (2,), (0, 1, 2)])
@pytest.mark.parametrize("shape", SHAPES[:4])
def test_step_of_misaligned_predictors(cuda_device, oracle, shape, which):
    import prj
    import workloads
    nx, ny, nz = shape
    Uh, Vh, Wh, yu, dx, dz = workloads.projection_inputs(nx, ny, nz, seed=62)
    dt, wall = 0.37, (0.01, 0.0, -0.02, 0.03, 0.0, 0.04)
    with prj.Plan.from_yu(nx, nz, dx, dz, yu, "consistent") as plan:
        hat = [to_dev(a) for a in (Uh, Vh, Wh)]
        hat = [_off(t) if i in which else t for i, t in enumerate(hat)]
        out = [empty_like_dev((nx + 2, nz + 2, ny + 2)) for _ in range(3)]
        P = empty_like_dev((nx, nz, ny))
        plan.projection_step(*hat, *out, P, dt, wall=wall)
        got = [from_dev(t) for t in (*out, P)]
    want = oracle.projection(Uh, Vh, Wh, dx, dz, dt, yu, "consistent", wall)
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= 1e-12 * np.abs(w).max()


def test_rank_lines_off_a_boundary_are_refused(cuda_device):
    import ctypes
    import torch
    import prj
    import workloads
    nx, ny, nz = 64, 8, 48
    _, yu, dx, dz = workloads.poisson_rhs(nx, ny, nz, seed=1)
    with prj.Plan(nx, nz, ny, dx, dz, prj.bands(yu, "consistent")) as plan:
        buf = torch.zeros(ny * nz * 4 * 2 + 2, dtype=torch.float64, device="cuda")
        rc = prj.load_library().prj_dist_thomas(plan.handle, ctypes.c_void_p(buf.data_ptr() + 8), 0, 4, None)
        assert rc == prj.PRJ_ERR_ARG

"""The z kernels that keep or share one x wavenumber over a cluster of CTAs, against the three
split kernels: the slab kernel (rows resident in shared memory) and the cluster form of the
per-wavenumber kernel.  Butterflies, tables and Thomas operation order are the same, so the
solves agree bit for bit; a requested row count (z_rows) keeps the split kernels.
"""
import numpy as np
import pytest

from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu


def _plan(nx, ny, nz):
    import prj
    import workloads
    yu = workloads.tanh_faces(ny)
    return prj.Plan(nx, nz, ny, 2 * np.pi / nx, np.pi / nz, prj.bands(yu, "consistent"))


def _solve(plan, rhs):
    t = to_dev(rhs)
    plan.poisson_fp64(t)
    plan.check_error()
    return from_dev(t)


def _both(nx, ny, nz, rhs, **tuning):
    """(default route with `tuning`, split kernels), and the default route's launches."""
    with _plan(nx, ny, nz) as plan:
        plan.set_tuning(**tuning)
        launches = plan.launches_per_step()
        got = _solve(plan, rhs)
    with _plan(nx, ny, nz) as plan:
        plan.set_tuning(z_mode=0, z_rows=4)
        assert plan.launches_per_step() == 6
        want = _solve(plan, rhs)
    return got, want, launches


def _rhs(nx, ny, nz, seed=0):
    return np.asfortranarray(np.random.default_rng(seed).uniform(-1, 1, (nx, nz, ny)))


# planes per CTA: one, a remainder of one, blocks of two and four cut short, a whole column;
# z lengths with a compile-time plan, with runtime radices, and no multiple of 8
@pytest.mark.parametrize("shape", [(32, 8, 16), (48, 33, 24), (30, 41, 64), (16, 64, 96), (20, 23, 50), (16, 30, 27),
                                   (24, 19, 384), (16, 16, 640)])
@pytest.mark.parametrize("planes", [0, 1, 3, 6, 13, 64])
def test_slab_equals_split(cuda_device, shape, planes):
    nx, ny, nz = shape
    if planes and (ny + min(planes, ny) - 1) // min(planes, ny) > 8:
        pytest.skip("more than eight CTAs per wavenumber")
    got, want, launches = _both(nx, ny, nz, _rhs(nx, ny, nz), z_planes=planes)
    if planes in (0, 6, 13) and nz <= 96:
        assert launches == 4  # one z kernel
    np.testing.assert_array_equal(got, want)


# threads without a line, and (270, 288) threads with a second line and without; half of the planes
# far below the division's window
@pytest.mark.parametrize("nz", [2, 9, 32, 96, 225, 250, 270, 288])
def test_slots_without_a_line(cuda_device, nz):
    nx, ny = 16, 24
    rhs = _rhs(nx, ny, nz, 4)
    rhs[:, :, : ny // 2] *= 2.0 ** -1000
    got, want, launches = _both(nx, ny, nz, rhs)
    assert launches == 4
    np.testing.assert_array_equal(got, want)


# clusters of two to eight CTAs, chunks cut short at the top, more wavenumbers than SMs
@pytest.mark.parametrize("shape", [(256, 128, 128), (256, 67, 128), (300, 130, 192), (200, 150, 256), (128, 97, 384),
                                   (330, 200, 64), (64, 130, 256), (150, 60, 96)])
def test_cluster_equals_split(cuda_device, shape):
    nx, ny, nz = shape
    got, want, launches = _both(nx, ny, nz, _rhs(nx, ny, nz, 1))
    assert launches == 4
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("shape", [(64, 40, 32), (256, 96, 128)])
@pytest.mark.parametrize("kind", ["zero", "2^-960", "2^-1010", "one plane", "infinite"])
def test_quotients_outside_the_window(cuda_device, shape, kind):
    """Zeros of both signs, quotients below 2^-900, subnormals, and infinities: the sweeps redo
    the planes concerned by plain division, as the split kernels do."""
    nx, ny, nz = shape
    rhs = _rhs(nx, ny, nz, 2)
    if kind == "zero":
        rhs[:] = 0.0
        rhs[::3] = -0.0
    elif kind == "one plane":
        rhs[:, :, 1:] = 0.0
    elif kind == "infinite":
        rhs[3, 5, 7] = np.inf
    else:
        rhs *= 2.0 ** int(kind[2:])
    got, want, _ = _both(nx, ny, nz, rhs)
    np.testing.assert_array_equal(got, want)
    if kind == "zero":
        assert not got.any()


@pytest.mark.parametrize("shape", [(14, 6, 7), (22, 9, 77), (26, 12, 143), (18, 8, 81), (20, 7, 100), (182, 10, 198),
                                   (360, 12, 250), (34, 9, 34), (62, 5, 46), (77, 9, 59), (98, 6, 121), (2, 8, 13),
                                   (770, 3, 130), (1690, 4, 26)])
def test_ragged_lengths(cuda_device, oracle, shape):
    """Radices 7, 9, 10, 11 and 13 of the runtime transforms, and lengths with larger primes,
    against the oracle within the parity bound of the other lengths."""
    import prj
    import workloads
    nx, ny, nz = shape
    rhs = _rhs(nx, ny, nz, 3)
    yu = workloads.tanh_faces(ny)
    b6 = prj.bands(yu, "reference")
    dx, dz = 2 * np.pi / nx, np.pi / nz
    with prj.Plan(nx, nz, ny, dx, dz, b6) as plan:
        got = _solve(plan, rhs)
    want, _ = oracle.poisson(rhs, dx, dz, b6)
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


def test_refused_lengths_stay_refused(cuda_device):
    """The mixed-precision solve and an explicit split z kernel take products of 2, 3 and 5 only."""
    import prj
    import torch
    for nx, nz in ((28, 32), (32, 28)):
        with _plan(nx, 8, nz) as plan:
            with pytest.raises(prj.PrjError):
                plan.poisson_mixed(torch.zeros((8, nz, nx), dtype=torch.float64, device=cuda_device))
            if nz == 28:
                assert plan.tuning["z_mode"] == 1
                with pytest.raises(prj.PrjError):
                    plan.set_tuning(z_mode=0)


def test_z_mode_names_the_kernels(cuda_device):
    """A z_mode that the caller gives is what runs, also where it is the plan's default; without
    one, other fields and a round trip through the plan's tuning keep the choice by size."""
    import prj
    nx, ny, nz = 48, 33, 24
    rhs = _rhs(nx, ny, nz, 5)
    with _plan(nx, ny, nz) as plan:
        t0 = plan.tuning
        assert t0["z_mode"] == 0 and t0["z_auto"] and plan.launches_per_step() == 4
        got = {"auto": _solve(plan, rhs)}
        plan.set_tuning(z_mode=0)
        assert plan.launches_per_step() == 6
        got["split"] = _solve(plan, rhs)
        plan.set_tuning(x_rows=4)
        assert plan.launches_per_step() == 6
        plan.set_tuning(**t0)
        assert plan.tuning == t0 and plan.launches_per_step() == 4
        plan.set_tuning(x_rows=4)
        assert plan.tuning["z_auto"] and plan.launches_per_step() == 4
        # the ABI: a tuning that was read and written back names the kernels it holds
        import ctypes
        t = prj.Tuning()
        lib = prj.load_library()
        assert lib.prj_plan_get_tuning(plan.handle, ctypes.byref(t)) == prj.PRJ_OK
        assert lib.prj_plan_set_tuning(plan.handle, ctypes.byref(t)) == prj.PRJ_OK
        assert plan.launches_per_step() == 6
        assert lib.prj_plan_set_z_auto(plan.handle, 1) == prj.PRJ_OK
        assert plan.launches_per_step() == 4
    np.testing.assert_array_equal(got["auto"], got["split"])
    with _plan(28, 9, 77) as plan:  # no in-place default: the fused kernel when named
        assert plan.tuning["z_mode"] == 1
        before = plan.launches_per_step()
        plan.set_tuning(z_planes=4)
        assert plan.launches_per_step() == 4
        plan.set_tuning(z_planes=0, z_mode=1)
        assert plan.launches_per_step() == 4 and not plan.tuning["z_auto"]
        plan.set_tuning(z_auto=True)
        assert plan.launches_per_step() == before
    # planes per CTA that would take more than one wave of clusters
    with _plan(400, 64, 64) as plan:
        assert plan.tuning["z_mode"] == 0
        plan.set_tuning(z_planes=8)
        assert plan.launches_per_step() == 6


# wavenumbers x CTAs that free SM slots would hold but the GPCs do not, long rows on chip, and
# k_zline below two wavenumbers per SM at long rows, each slower than the three kernels; clusters of
# four where more would also be resident; short chains of long rows
@pytest.mark.parametrize("shape,launches", [((32, 68, 768), 6), ((32, 256, 240), 6), ((32, 384, 160), 6),
                                            ((36, 83, 600), 6), ((32, 64, 640), 6), ((300, 24, 1536), 6),
                                            ((300, 100, 1024), 6), ((96, 300, 256), 4), ((48, 105, 384), 4),
                                            ((32, 400, 384), 4), ((96, 53, 384), 6), ((384, 36, 512), 6),
                                            ((384, 66, 512), 4)])
def test_routes_where_a_second_wave_would_run(cuda_device, shape, launches):
    nx, ny, nz = shape
    got, want, n = _both(nx, ny, nz, _rhs(nx, ny, nz, 6))
    assert n == launches
    np.testing.assert_array_equal(got, want)

"""GPU tests of the device-side failure paths, made to happen without faulting
the GPU: every wait that runs out is bounded and reports a status, after which
the same process keeps sorting and simulating correctly.

* The radix sort's decoupled look-back waits on a predecessor tile that never
  publishes (its ticket is taken before the pass starts): the bounded wait
  gives up and the call returns MPM_ERR_TIMEOUT.
* The look-back status words of the radix sort and of the block scan carry a
  30-bit epoch: sorts across its wrap stay bit-exact against a CPU stable sort.
* The FP64 SVD (the reference's unbounded implicit-shift QR,
  Core/Matrices/MATRIX_3X3.cpp:202-236) gets a one-sweep bound: the substep
  reports MPM_ERR_NOT_CONVERGED.
* Each of the library's device allocations reports, once, that memory is short
  (a failure made on the host): the call returns MPM_ERR_NOMEM and leaves nothing
  half-built behind, so the same call works when it is made again.
The reference's counterparts are assertion failures that throw
(Core/Log/DEBUG_UTILITIES.cpp:95-103); here they are status codes.
"""
import numpy as np
import pytest

from physbam_b200 import scenes as S

pytestmark = pytest.mark.gpu

TIMEOUT, NOMEM, STATE, NOT_CONVERGED = 5, 6, 7, 8


def D():
    from physbam_b200 import driver
    return driver


def test_sort_lookback_timeout_is_reported(cuda_device):
    L = D().load_library()
    rng = np.random.default_rng(3)
    keys = rng.integers(0, 1 << 16, 10_000, dtype=np.uint32)
    rc = L.mpm_debug_sort_stall(keys.ctypes.data, keys.size, 16, 1024)
    assert rc == TIMEOUT
    # the context is still usable: a normal sort right after is bit-exact
    sk, perm = D().radix_sort_u32(keys, 16)
    ref = np.argsort(keys, kind="stable").astype(np.uint32)
    np.testing.assert_array_equal(perm, ref)
    np.testing.assert_array_equal(sk, keys[ref])


def test_sort_across_epoch_wrap(cuda_device):
    scene = S.small_3d(nsteps=8)
    drv = D().MPM_DRIVER(scene)
    drv.set_scene_particles(scene)
    drv._check(drv.L.mpm_debug_set_sort_epoch(drv.h, (1 << 30) - 3), "mpm_debug_set_sort_epoch")
    for it in range(6):
        if it % 2 == 0:
            drv.set_scene_particles(scene)     # a full sort of freshly uploaded keys next
        drv.Particle_To_Grid()
        keys, sk, perm = drv.sort_state()
        ref = np.argsort(keys >> 6, kind="stable").astype(np.uint32)
        np.testing.assert_array_equal(perm, ref, err_msg="sort %d" % it)
        np.testing.assert_array_equal(sk, keys[ref])
        drv.Apply_Forces()
        drv.Grid_To_Particle()
    drv.synchronize()
    drv.close()


@pytest.mark.parametrize("path", ["plain", "fast"])
def test_svd_non_convergence_is_reported(cuda_device, path):
    L = D().load_library()
    scene = S.small_3d(nsteps=2)
    if path == "fast":         # inverted F takes the FP64 SVD route on the fast path
        F = scene.F.copy()
        F[::3, :, 0] *= -1.0
        scene.F = F
    prec, p = (D().FP64, D().PATH_PLAIN) if path == "plain" else (D().FP32, D().PATH_FAST)
    assert L.mpm_debug_set_svd_iterations(1) == 0
    try:
        drv = D().MPM_DRIVER(scene, precision=prec, path=p)
        drv.set_scene_particles(scene)
        drv.Advance_One_Time_Step()
        with pytest.raises(D().MPMError) as e:
            drv.synchronize()
        assert e.value.code == NOT_CONVERGED
        drv.close()
    finally:
        assert L.mpm_debug_set_svd_iterations(64) == 0
    drv = D().MPM_DRIVER(scene, precision=prec, path=p)
    drv.set_scene_particles(scene)
    drv.advance(2)
    drv.synchronize()
    assert drv.count_valid() == scene.n
    drv.close()


def refuse_each(make, call, after=lambda drv: None):
    """`call(drv)` on a new handle per allocation it makes, that allocation refused: it returns
    MPM_ERR_NOMEM, and the same call made again works.  Its results, the undisturbed call's last."""
    out = []
    for k in range(1, 100):
        drv = make()
        drv._check(drv.L.mpm_debug_fail_allocation(drv.h, k), "mpm_debug_fail_allocation")
        try:
            try:
                out.append(call(drv))
                return out
            except D().MPMError as e:
                assert e.code == NOMEM, e
            after(drv)
            out.append(call(drv))
        finally:
            drv.close()
    raise AssertionError("never succeeded")


@pytest.mark.parametrize("G", [16, 40])                # dense node passes, listed tiles
@pytest.mark.parametrize("budget", [-1, 0])            # the whole tape, segments
@pytest.mark.parametrize("phase", ["forward", "backward"])
def test_rollout_short_of_memory(cuda_device, G, budget, phase):
    import torch
    scene = S.small_3d(G=G, ppc=1, with_walls=False)
    one = [torch.ones((scene.n, k), dtype=torch.float64, device="cuda") for k in (3, 3, 9, 9)]

    def make():
        drv = D().MPM_DRIVER(scene, precision=D().FP64, path=D().PATH_PLAIN)
        drv.set_diff_tape_budget(budget)
        drv.set_scene_particles(scene)
        if phase == "backward":
            drv.diff_forward(7, 3)
        return drv

    def call(drv):
        if phase == "forward":
            drv.diff_forward(7, 3)
            return [drv.get_particles()["X"]]
        return [g.cpu().numpy() for g in drv.diff_backward(*one)]

    out = refuse_each(make, call)
    slots = 6 if G == 16 else 8
    assert len(out) - 1 == (4 if phase == "forward" else 7) + (slots if (phase == "forward") == (budget < 0) else 0)
    for got in out[:-1]:
        for a, b in zip(got, out[-1]):
            assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()


def test_implicit_short_of_memory(cuda_device):
    scene = S.small_3d_implicit(nsteps=2)

    def make():
        drv = D().MPM_DRIVER(scene, precision=D().FP64, path=D().PATH_PLAIN)
        drv.set_scene_particles(scene)
        return drv

    def call(drv):
        drv.Advance_One_Time_Step()
        return drv.get_particles()["X"]

    out = refuse_each(make, call)
    assert len(out) >= 14
    for X in out[:-1]:
        assert np.abs(X - out[-1]).max() < 2e-9        # Newton to its own tolerance


@pytest.mark.parametrize("path,scene", [("plain", S.small_3d(G=40, ppc=1)), ("plain", S.small_snow_3d()),
                                        ("fast", S.small_3d()), ("fast", S.small_snow_3d())])
def test_upload_short_of_memory(cuda_device, path, scene):
    """More particles than the handle held: refused, it holds none and says so."""
    precision, path = (D().FP64, D().PATH_PLAIN) if path == "plain" else (D().FP32, D().PATH_FAST)

    def make():
        drv = D().MPM_DRIVER(scene, precision=precision, path=path)
        drv.set_scene_particles(scene.subset(np.arange(100)))
        drv.advance(2)
        return drv

    def call(drv):
        drv.set_scene_particles(scene)
        drv.advance(3)
        drv.synchronize()
        return drv.get_particles()["X"]

    def refused(drv):
        with pytest.raises(D().MPMError) as e:
            drv.advance(1)
        assert e.value.code == STATE

    out = refuse_each(make, call, refused)
    assert len(out) >= 10
    for X in out[:-1]:
        assert np.abs(X - out[-1]).max() < (1e-12 if precision == D().FP64 else 2e-6)

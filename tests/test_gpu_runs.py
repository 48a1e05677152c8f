"""GPU tests of the kernels that sum runs of particles and visit lists of grid tiles, at the
sizes where they can go wrong, against the C oracle.

* Particle counts around a warp (plain, adjoint and implicit scatters), a work item and a
  block (fast P2G and G2P, every launch shape), in shuffled order, some invalid, one without
  mass.
* Grids past the size from which the plain path lists the tiles that P2G touched: explicit and
  implicit substeps, a rollout recorded in place.
* The hand-over and read-back of particles, and Compute_Dt's speed bound, around a warp.

Tolerances: FP64 sums of at most 27 x 60 terms in another order, some 1e-13 of the largest
value, over ten substeps; FP32 as in test_gpu_parity.py.
"""
import ctypes

import numpy as np
import pytest

import oracle
from physbam_b200 import scenes as S

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 31, 33, 97, 257]


def D():
    from physbam_b200 import driver
    return driver


def pick(scene, n, seed=3):
    """n particles of the scene in no order at all."""
    return scene.subset(np.random.default_rng(seed).permutation(scene.n)[:n])


def run_oracle(scene, steps, valid=None):
    st = oracle.State(scene)
    if valid is not None:
        st.valid[:] = valid
    oracle.run(st, steps)
    return st


def run_gpu(scene, steps, precision, path, valid=None, shape=None):
    drv = D().MPM_DRIVER(scene, precision=precision, path=path)
    if shape is not None:
        drv.set_launch_shape(*shape)
    drv.set_particles(scene.X, scene.V, scene.F, scene.B, scene.mass, scene.volume, scene.mu, scene.lam, valid=valid)
    drv.advance(steps)
    drv.synchronize()
    got = drv.get_particles()
    drv.close()
    return got


def check(got, st, tol):
    keep = st.valid.astype(bool)
    np.testing.assert_array_equal(got["valid"], keep)
    vmax = max(np.abs(st.V).max(), 1e-12)
    for k, ref, scale in (("X", st.X, 1.0), ("V", st.V, vmax), ("F", st.F_rowmajor(), 1.0),
                          ("B", st.B_rowmajor(), vmax / st.scene.dx)):
        assert np.abs(got[k] - ref)[keep].max() <= tol[k] * scale, k


TOL64 = {"X": 1e-12, "V": 1e-9, "F": 1e-10, "B": 1e-8}
TOL32 = {"X": 2e-6, "V": 2e-3, "F": 1e-4, "B": 2e-3}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", COUNTS)
def test_plain_scatter_counts(cuda_device, dim, n):
    scene = pick(S.small_2d() if dim == 2 else S.small_3d(), n)
    valid = np.ones(scene.n, np.uint8)
    valid[::5] = 0
    if n < 3:
        valid[:] = 1
    check(run_gpu(scene, 10, D().FP64, D().PATH_PLAIN, valid), run_oracle(scene, 10, valid), TOL64)


@pytest.mark.parametrize("variant,threads", [(0, 64), (1, 256), (2, 64), (3, 128), (0, 256), (3, 64)])
@pytest.mark.parametrize("n", [1, 63, 65, 127, 129, 257, 600])
def test_fast_item_counts(cuda_device, variant, threads, n):
    """All particles in one block and its neighbours: items of every size up to the largest."""
    base = S.small_3d()
    scene = pick(base, n)
    h = 1.0 / 16
    rng = np.random.default_rng(n)
    scene.X[:] = 0.25 + 0.05 * h + rng.random((scene.n, 3)) * np.array([0.9, 0.9, 3.9]) * h
    scene.mass[-1] *= 1e-3
    check(run_gpu(scene, 10, D().FP32, D().PATH_FAST, shape=(variant, threads, 1)), run_oracle(scene, 10), TOL32)


def test_fast_block_of_many_items(cuda_device):
    """4,500 particles in one block: more work items (64 particles each) than a warp has lanes."""
    scene = pick(S.small_3d(ppc=24), 4500)
    scene.X[:] = 0.25 + (0.1 + 3.8 * np.random.default_rng(1).random((scene.n, 3))) / 16
    assert scene.n == 4500
    check(run_gpu(scene, 5, D().FP32, D().PATH_FAST, shape=(2, 64, 1)), run_oracle(scene, 5), TOL32)


def test_fast_particle_without_mass(cuda_device):
    """A particle of zero mass takes part with its force alone, as on the plain path."""
    scene = pick(S.small_3d(), 700)
    scene.mass[::50] = 0.0
    check(run_gpu(scene, 5, D().FP32, D().PATH_FAST), run_oracle(scene, 5), TOL32)


@pytest.mark.parametrize("upload", [False, True])
def test_fast_force_on_massless_nodes(cuda_device, upload):
    """The force of a stressed particle of zero mass away from the others is gone with its substep: a
    body that reaches its nodes later, in the same run or after a re-upload, moves as on the plain path."""
    scene = pick(S.small_3d(with_walls=False, friction=0.0), 400)
    scene.X[:] = 0.3 + 0.2 * np.random.default_rng(4).random((scene.n, 3))
    scene.V[:] = [20.0, 0.0, 0.0]
    scene.X[-8:] = [0.72, 0.4, 0.4]                # three cells ahead of the body
    scene.V[-8:] = 0.0
    scene.mass[-8:] = 0.0
    scene.F[-8:] = np.diag([0.5, 1.2, 0.9])
    later = scene.copy()
    later.X[:-8, 0] += 0.2
    out = []
    for precision, path in ((D().FP32, D().PATH_FAST), (D().FP64, D().PATH_PLAIN)):
        drv = D().MPM_DRIVER(scene, precision=precision, path=path)
        drv.set_scene_particles(scene)
        drv.advance(40 if upload else 100)         # short of the massless ones' nodes, or over them
        if upload:
            drv.set_scene_particles(later)
            drv.advance(20)
        drv.synchronize()
        out.append(drv.get_particles())
        drv.close()
    got, ref = out
    assert ref["X"][:-8, 0].max() > 0.62           # within a cell and a half of the massless ones
    # positions: the velocities' tolerance over 100 substeps of 1e-4 (left-over forces: 3e-2)
    vmax = np.abs(ref["V"]).max()
    assert np.abs(got["V"] - ref["V"])[:-8].max() <= 2e-3 * vmax
    assert np.abs(got["X"] - ref["X"])[:-8].max() <= 100 * 1e-4 * 2e-3 * vmax


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("field,bad", [("V", np.nan), ("V", np.inf), ("B", -np.inf), ("F", np.nan), ("mass", np.inf),
                                       ("mass", np.nan), ("V", 1e37)])
def test_fast_p2g_reports_non_finite(cuda_device, variant, field, bad):
    """A particle that is not finite, or whose momentum is not, is reported by the P2G phase already
    and leaves the grid finite."""
    scene = pick(S.small_3d(), 600)
    getattr(scene, field)[300] = bad
    if bad == 1e37:
        scene.mass[300] = 1e6
    drv = D().MPM_DRIVER(scene)
    drv.set_launch_shape(variant, 128, 1)
    drv.set_scene_particles(scene)
    drv.Particle_To_Grid()
    with pytest.raises(D().MPMError) as e:
        drv.synchronize()
    assert e.value.code == 3
    drv.Apply_Forces()
    grid = drv.get_grid()
    drv.close()
    assert (grid["grid_m"] > 0).sum() > 100
    assert all(np.isfinite(grid[k]).all() for k in grid)


@pytest.mark.parametrize("shape", [(3, 128, 1), (2, 64, 1), (1, 256, 1), (3, 64, 1), (3, 128, 2), (0, 128, 1)])
def test_fast_many_items_in_two_scenes(cuda_device, shape):
    """Enough work items that G2P streams them (two and more per CTA), blocks of every fill, a
    scene change on the way, walls with friction, particles that leave the domain: against the
    plain path in FP64, scene by scene."""
    scenes = [S.small_3d(G=88, friction=0.3), S.small_3d(seed=9, G=82, model=S.NEO_HOOKEAN, with_walls=False)]
    keep = np.random.default_rng(2).random(scenes[1].n) < 0.6
    scenes[1] = scenes[1].subset(np.flatnonzero(keep))
    scenes[1].X[:50] = 1.0 - 1e-6
    scenes[1].V[:50] = 10.0
    drv = D().MPM_BATCH(scenes)
    drv.set_launch_shape(*shape)
    drv.set_scene_particles()
    drv.advance(4, 1e-5)
    drv.synchronize()
    streamed = ctypes.c_int()
    drv._check(drv.L.mpm_debug_g2p_streamed(drv.h, ctypes.byref(streamed)), "mpm_debug_g2p_streamed")
    assert streamed.value == 1
    got = drv.split(drv.get_particles())
    drv.close()
    for s, g in zip(scenes, got):
        ref = D().MPM_DRIVER(s, precision=D().FP64, path=D().PATH_PLAIN)
        ref.set_scene_particles(s)
        ref.advance(4, 1e-5)
        r = ref.get_particles()
        ref.close()
        np.testing.assert_array_equal(g["valid"], r["valid"])
        keep, vmax = r["valid"].astype(bool), np.abs(r["V"]).max()
        for k, scale in (("X", 1.0), ("V", vmax), ("F", 1.0), ("B", vmax / s.dx)):
            assert np.abs(g[k] - r[k])[keep].max() <= TOL32[k] * scale, k


@pytest.mark.parametrize("ppc", [1, 8])
def test_fast_grid_of_one_sum_per_node(cuda_device, ppc):
    """More than 2^28 nodes (P2G keeps one sum per node, not four): a body in the corner of a 660^3
    grid moves as on a 40^3 grid of the same cells."""
    scene = S.small_3d(G=40, ppc=ppc, with_walls=False)
    far = scene.copy()
    far.counts = [660] * 3
    far.domain_max = [660 / 40.0] * 3
    got, ref = (run_gpu(s, 10, D().FP32, D().PATH_FAST) for s in (far, scene))
    np.testing.assert_array_equal(got["valid"], ref["valid"])
    vmax = np.abs(ref["V"]).max()
    for k, scale in (("X", 1.0), ("V", vmax), ("F", 1.0), ("B", vmax / scene.dx)):
        assert np.abs(got[k] - ref[k]).max() <= TOL32[k] * scale, k


@pytest.mark.parametrize("G", [16, 40])
def test_plain_captured_substeps_after_upload(cuda_device, G):
    """Captured substeps kept over an upload of as many particles run on the new ones; an upload of
    another number, new objects and another step are captured anew."""
    scene = S.small_3d(G=G, ppc=2)
    other = scene.copy()
    other.X += 0.01
    other.V *= -0.5
    other.mu *= 2.0
    few = other.subset(np.arange(other.n - 50))
    bare = scene.copy()
    bare.objects = []
    drv = D().MPM_DRIVER(scene, precision=D().FP64, path=D().PATH_PLAIN)
    for s, steps, dt in ((scene, 4, 1e-4), (other, 4, 1e-4), (few, 4, 1e-4), (scene, 3, 5e-5), (bare, 3, 5e-5)):
        if s is bare:
            drv.set_collision_objects([])
        drv.set_scene_particles(s)
        drv.advance(steps, dt)
        drv.synchronize()
        ref = s.copy()
        ref.dt = dt
        check(drv.get_particles(), run_oracle(ref, steps), TOL64)
    drv.close()


def big(scene_fn, **kw):
    """A small body on a 40^3 grid: 46^3 nodes, past the size from which tiles are listed."""
    return scene_fn(G=40, **kw)


@pytest.mark.parametrize("n", [1, 97, 3000])
def test_plain_listed_tiles(cuda_device, n):
    scene = pick(big(S.small_3d, ppc=4), n)
    check(run_gpu(scene, 10, D().FP64, D().PATH_PLAIN), run_oracle(scene, 10), TOL64)


@pytest.mark.parametrize("G", [156, 164, 330])
def test_plain_tile_list_of_large_grids(cuda_device, G):
    """The list of touched tiles around the sizes where it takes a count first (128 spans of 32,768 nodes)
    and where a CTA takes several spans (1,024): bodies in the low and the high corner of the grid
    move as on a small grid of the same cells."""
    scene = S.small_3d(G=24, ppc=2, with_walls=False)
    ref = run_gpu(scene, 5, D().FP64, D().PATH_PLAIN)
    grid = scene.copy()
    grid.counts, grid.domain_max = [G] * 3, [G / 24.0] * 3
    grid = grid.subset(np.tile(np.arange(scene.n), 2))
    shift = (G - 24) // 8 * 8 / 24.0                 # whole cells, exact in binary
    grid.X[scene.n:] += shift
    got = run_gpu(grid, 5, D().FP64, D().PATH_PLAIN)
    # a position is rounded at the size of the shift, and B divides that by dx twice
    eps, vmax = 2.0 ** -52 * (1 + shift), np.abs(ref["V"]).max()
    for body in (0, 1):
        part = slice(body * scene.n, (body + 1) * scene.n)
        assert np.abs(got["X"][part] - body * shift - ref["X"]).max() <= 100 * eps
        assert np.abs(got["V"][part] - ref["V"]).max() <= 1e-9 * vmax


def test_plain_node_passes_before_p2g(cuda_device):
    """The phase entry points in any order: node passes before the first P2G find an empty tile
    list; forces of particles that have moved since the last P2G leave nothing on the grid for
    the next; a grid update after the reflection was switched off runs over the whole grid."""
    scene = pick(big(S.small_3d, ppc=4), 500)
    drv = D().MPM_DRIVER(scene, precision=D().FP64, path=D().PATH_PLAIN)
    drv.set_scene_particles(scene)
    drv.add_grid_forces(np.ones(tuple(c + 2 * S.GHOST for c in scene.counts) + (3,)))
    drv.Apply_Forces()
    drv.advance(3)
    drv.Apply_Forces()
    drv.advance(2)
    drv.synchronize()
    check(drv.get_particles(), run_oracle(scene, 5), TOL64)
    grids = []
    for reflect in (False, True):                  # far from the faces reflection changes nothing
        drv.set_scene_particles(scene)
        if reflect:
            drv.set_reflection(S.Reflection(side_type=(S.BC_SLIP,) * 6))
        drv.Particle_To_Grid()
        if reflect:
            drv.set_reflection(None)
        drv.Apply_Forces()
        grids.append(drv.get_grid())
    drv.close()
    assert np.abs(grids[0]["grid_v"]).max() > 0
    for k in grids[0]:
        np.testing.assert_allclose(grids[1][k], grids[0][k], rtol=0, atol=1e-12 * np.abs(grids[0][k]).max())


def test_plain_tiles_of_moving_bodies(cuda_device):
    """Two bodies, their particles in no order, that part and on their way cross several tiles and
    leave others (up to five cells per axis)."""
    scene = pick(big(S.small_3d, ppc=2, with_walls=False), 1500)
    half = scene.n // 2
    scene.X[:, 0] = 0.24 + 0.4 * (scene.X[:, 0] - 0.2)
    scene.X[:half, 0] += 0.36                          # 0.24 to 0.4, and 0.6 to 0.76
    scene.V[:half] = [30.0, 10.0, 20.0]
    scene.V[half:] = [-30.0, 10.0, -20.0]
    check(run_gpu(scene, 40, D().FP64, D().PATH_PLAIN), run_oracle(scene, 40), TOL64)


def test_implicit_listed_tiles(cuda_device):
    """On a grid with listed tiles, over a sticking floor: the solve agrees with itself to the
    Newton tolerance and, at a small step, with the explicit substep.  Backward and symplectic
    Euler differ by (dt omega)^2 of the velocity per step, omega^2 = 12 (c / h)^2 the grid's
    highest."""
    dt = 2e-5
    scene = S.small_3d(G=40, with_walls=False, dt=dt)
    scene.objects = S.walls(3, scene.counts, scene.domain_min, scene.domain_max, 1 << 3, S.STICK, 0.0, 0.15)
    st = run_oracle(scene, 2)
    scene.implicit = S.Implicit()
    got = run_gpu(scene, 2, D().FP64, D().PATH_PLAIN)
    again = run_gpu(scene, 2, D().FP64, D().PATH_PLAIN)
    vmax = np.abs(st.V).max()
    assert np.abs(got["X"] - again["X"]).max() < 2e-9 and np.abs(got["V"] - again["V"]).max() < 1e-6 * vmax
    c = np.sqrt((scene.lam + 2 * scene.mu).max() * scene.volume[0] / scene.mass[0])
    assert np.abs(got["V"] - st.V).max() < 2 * 12 * (dt * c / scene.dx) ** 2 * vmax


@pytest.mark.parametrize("G,budget", [(16, -1), (16, 0), (40, -1), (40, 0)])
def test_recorded_rollout_state(cuda_device, G, budget):
    """The rollout's G2P writes from one tape slot to the next; the particles it ends with are
    those of the plain substeps, frozen and leaving ones among them, with the tape whole or in
    segments, and a backward pass leaves them there."""
    import torch
    scene = S.small_3d(G=G, ppc=2, with_walls=False)
    scene.X[:7] = 1.0 - 1e-5                       # leave in the first substeps
    scene.V[:7] = 5.0
    st = run_oracle(scene, 11)
    drv = D().MPM_DRIVER(scene, precision=D().FP64, path=D().PATH_PLAIN)
    drv.set_diff_tape_budget(budget)
    drv.set_scene_particles(scene)
    drv.diff_forward(11, 4)
    check(drv.get_particles(), st, TOL64)
    one = [torch.ones((scene.n, k), dtype=torch.float64, device="cuda") for k in (3, 3, 9, 9)]
    g = drv.diff_backward(*one)
    check(drv.get_particles(), st, TOL64)
    assert all(bool(torch.isfinite(x).all()) for x in g)
    drv.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", COUNTS)
def test_hand_over_and_back(cuda_device, n, dtype):
    """Particles come back as they went in (rounded to float), in the caller's order, after a
    substep of no length to speak of has sorted them; the speed bound equals the totals'."""
    scene = pick(S.small_3d(), n)
    drv = D().MPM_DRIVER(scene)
    drv.set_scene_particles(scene, dtype=dtype)
    got = drv.get_particles(dtype=dtype)
    for k in ("X", "V", "F", "B"):
        np.testing.assert_array_equal(got[k], getattr(scene, k).astype(np.float32).astype(dtype))
    drv.advance(1, 1e-12)
    got = drv.get_particles(dtype=dtype)
    np.testing.assert_allclose(got["X"], scene.X, atol=1e-6)
    v = drv.particle_totals()["max_affine_speed"]
    assert drv.compute_dt(cfl=1e-3, max_dt=1e3) == pytest.approx(1e-3 * scene.dx / v, rel=1e-15)
    drv.close()

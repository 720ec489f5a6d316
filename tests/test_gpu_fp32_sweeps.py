"""The FP32 sweeps' team variants on scenes built for them: single triangles standing on a fixed ground, each with one
contact, so that a scene's contacts, levels and touched bodies are known before it is stepped."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chips(count, side=None, spacing=0.6):
    """`count` bodies of one triangle each, a tip pressed into the ground, in rows on a square (scene arrays).  A chip's
    grid is smaller than twice the margin inside which the search takes contacts, so only its tip makes one."""
    from rainbow_b200 import api as API, engine_io
    from rainbow_b200.types import Grid
    side = side or int(np.ceil(np.sqrt(count)))
    engine = API.create_engine("cuda:0")
    engine.params.resolution = 12
    API.create_surfaces_interaction(engine, "m", "m", 0.0, np.array([0.5, 0.5, 0.5]))
    API.create_gravity_force(engine, "gravity", 9.81, np.array([0.0, 1.0, 0.0]))
    V, T = API.create_box(spacing * side + 8.0, 1.0, spacing * side + 8.0)
    API.create_shape(engine, "ground", API.create_mesh(V, T))
    API.create_rigid_body(engine, "ground")
    API.connect_shape(engine, "ground", "ground")
    API.set_position(engine, "ground", np.array([0.0, -0.5, 0.0]), True)
    API.set_orientation(engine, "ground", np.array([1.0, 0.0, 0.0, 0.0]), True)
    API.set_body_type(engine, "ground", "fixed")
    API.set_mass_properties(engine, "ground", 1.0)
    API.set_body_material(engine, "ground", "m")
    a = {k: (v.cpu().numpy() if hasattr(v, "cpu") else v) for k, v in engine_io.scene_arrays(engine).items()}
    tip = np.array([[0.0, -0.2, 0.01], [0.2, 0.1, 0.02], [-0.2, 0.15, -0.03]])
    meta = Grid(tip.min(0) - 0.1, tip.max(0) + 0.1, 3, 3, 3).meta()
    for key, v in (("shape_V", tip), ("shape_T", np.array([[0, 1, 2]], np.int32)), ("shape_grid", np.ones(27)),
                   ("shape_grid_meta", np.reshape(meta, (1, 12)))):
        a[key] = np.concatenate([a[key], v])
    for key, n in (("shape_v_off", 3), ("shape_t_off", 1), ("shape_g_off", 27)):
        a[key] = np.append(a[key], a[key][-1] + n)
    rng = np.random.default_rng(1)   # a chip's state depends on its number alone
    i = np.arange(count)
    place = np.stack([spacing * (i % side - side / 2), 0.19 + 0.005 * rng.random(count), spacing * (i // side - side / 2)], 1)
    more = dict(body_shape=np.ones(count, np.int32), body_r=place, body_q=np.tile([1.0, 0.0, 0.0, 0.0], (count, 1)),
                body_v=rng.uniform([-1.0, -2.0, -1.0], [1.0, -1.0, 1.0], (count, 3)), body_w=rng.uniform(-2.0, 2.0, (count, 3)),
                body_mass=rng.uniform(0.5, 3.0, count), body_inertia=rng.uniform(0.01, 0.1, (count, 3)),
                body_fixed=np.zeros(count, np.uint8), body_material=np.zeros(count, np.int32),
                body_force_order=np.zeros((count, a["body_force_order"].shape[1]), np.int32))
    for key, v in more.items():
        a[key] = np.concatenate([a[key], v])
    return a


def step(arrays, sweeps, precision="fp32", interval=4, **launch):
    """One step of `sweeps` sweeps with a tolerance that is never met: (velocities, statistics, impulses)."""
    from rainbow_b200 import world as W
    w = W.DeviceWorld([arrays], device="cuda:0", max_iterations=max(sweeps, 1))
    rp = W.make_rb_params(W.params_from_vector(arrays["params"]), termination="residual_fixed_r",
                          residual_tolerance=-1.0, residual_interval=interval, precision=precision)
    rp.max_iterations = sweeps
    for key, v in launch.items():
        setattr(rp, key, v)
    assert w.step(rp) == 0
    return w.state()[1], w.stats()[0], w.contacts()["sol"].reshape(-1, 4)


@pytest.mark.parametrize("count", [1, 2, 7, 8])
def test_sweeps_of_one_step(count):
    """Every body with one contact: a sweep is one step, and the next one starts from the impulses that the same lanes
    have just stored.  Up to eight contacts a quad of lanes takes each; with nine a lane does, for the first ones with
    the same operands in the same order, so the velocities are the same to the bit.  Against FP64 after as many sweeps:
    twelve sweeps of ~60 FP32 operations, 12 x 60 x 2^-24 = 4e-5 of the largest value."""
    quads, lanes = chips(count, side=3), chips(9, side=3)
    for key in lanes:   # the first bodies of both are the same
        if key.startswith("body_"):
            quads[key] = lanes[key][:count + 1]
    u, st, sol = step(quads, 12)
    assert (st.n_contacts, st.n_levels, st.fp32_sweeps) == (count, 1, 12)
    u9, st9, sol9 = step(lanes, 12)
    assert (st9.n_contacts, st9.n_levels, st9.fp32_sweeps) == (9, 1, 12)
    np.testing.assert_array_equal(sol, sol9[:count])
    np.testing.assert_array_equal(u, u9[:count + 1])
    u64, _, sol64 = step(quads, 12, precision="fp64")
    assert np.abs(sol[:, 1:]).max() > 0.0   # friction is at work
    np.testing.assert_allclose(sol, sol64, rtol=0.0, atol=4e-5 * np.abs(sol64).max())
    np.testing.assert_allclose(u, u64, rtol=0.0, atol=4e-5 * np.abs(u64).max())


@pytest.mark.parametrize("interval", [1 << 30, (1 << 31) - 1])
def test_residual_intervals_beyond_the_sweeps(interval):
    """A residual test spaced further than the sweeps of a step can go, up to the largest number the parameter holds, is
    made at their end only: the same bits as any interval beyond the cap."""
    a = chips(20)
    u, st, sol = step(a, 40, interval=interval)
    u1, st1, sol1 = step(a, 40, interval=1000)
    assert st.fp32_sweeps == st1.fp32_sweeps == 40 and st.n_contacts == 20
    np.testing.assert_array_equal(sol, sol1)
    np.testing.assert_array_equal(u, u1)


def test_profiled_steps_run_the_contact_search_of_the_others():
    """Profiling alone does not change the kernels that are timed: an FP32 step searches the FP64 grids, with as many
    lookups as the FP64 step's, and a world holds no FP32 copy of its grids.  Bit 2 asks for the check, which makes it."""
    from rainbow_b200 import world as W
    a = chips(20)
    w = W.DeviceWorld([a], device="cuda:0", max_iterations=200)
    x0, u0 = w.state()
    seen = []
    for precision, profiling in (("fp64", 1), ("fp32", 0), ("fp32", 1), ("fp32", 3)):
        assert not w.rb_shapes.grid32
        w.set_state(x0, u0)
        assert w.step(W.make_rb_params(W.params_from_vector(a["params"]), precision=precision, profiling=profiling,
                                       termination="residual_fixed_r")) == 0
        st = w.stats()[0]
        seen.append((st.n_grid_lookups, st.n_grid_lookups32, st.n_contacts))
    assert seen[0] == seen[2] and seen[0][0] > 0 and seen[1] == (0, 0, 20)
    assert seen[3][1] > 0 and w.rb_shapes.grid32


@pytest.mark.parametrize("count,scheme", [(40, "rigid_gauss_seidel"), (40, "parallel_jacobi"), (600, "rigid_gauss_seidel"),
                                          (1500, "rigid_gauss_seidel")])
@pytest.mark.parametrize("precision", ["fp32", "fp32_refine"])
def test_a_nan_impulse_is_never_reported_as_a_residual(count, scheme, precision):
    """One body with a NaN velocity among others: a NaN in its contact's impulses, whichever lanes and warps test it, makes
    the residual NaN and is no convergence.  (FP32 Gauss-Seidel sweeps leave one in the friction rows; a Jacobi sweep and
    the FP64 prox put zero there.)"""
    from rainbow_b200 import _native as N, world as W
    a = chips(count)
    out = []
    for bad in (False, True):
        a = dict(a, body_v=a["body_v"].copy())
        if bad:
            a["body_v"][3] = np.nan
        w = W.DeviceWorld([a], device="cuda:0", max_iterations=24)
        rp = W.make_rb_params(W.params_from_vector(a["params"]), termination="residual_fixed_r", residual_tolerance=1e-6,
                              residual_interval=4, precision=precision, scheme=scheme)
        rp.max_iterations = 24
        assert w.step(rp) == (N.STATUS_NONFINITE if bad else 0)
        out.append((w.stats()[0], w.contacts()["sol"].reshape(-1, 4)))
    (good_st, good), (bad_st, bad) = out
    assert bad_st.n_contacts == good_st.n_contacts > count // 2
    assert np.isfinite(good).all() and np.isfinite(good_st.residual)
    assert np.isnan(bad).any(axis=1).sum() == (precision == "fp32" and scheme == "rigid_gauss_seidel")
    if np.isnan(bad).any():
        assert np.isnan(bad_st.residual) and bad_st.exitcode == 0
    else:
        np.testing.assert_array_equal(bad[2], 0.0)

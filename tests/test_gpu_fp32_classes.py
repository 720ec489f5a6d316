"""The FP32 phase's size classes on one problem: a small pile solved by a warp from a slab, by a block from a slab, and,
with single triangles on a ground of their own far away added to its scene, from L2 through the ring, from L2 directly
and with the body records in L2 too.  The pile's contacts come first in every scene and share no body with the others,
so each class has to give them the same impulses, to the bit."""
import numpy as np
import pytest

from test_gpu_fp32_sweeps import chips

pytestmark = pytest.mark.gpu
SLAB, RING = 224 * 1024, 6 * 32 * 192


def size_class(K, nb, mid_slab=56 * 1024):
    """Which arrays of a scene of K contacts and nb bodies are on chip: contact rows of 208 bytes with 14 bytes of indices,
    64 bytes for each body a contact can touch, in 16-byte pieces."""
    up = lambda v: (v + 15) // 16 * 16  # noqa: E731
    nr = min(nb, 2 * K)
    bodies, lists = up(64 * nr), up(4 * K) + up(2 * (nr + 1))
    whole = up(208 * K) + up(2 * K) + up(8 * K) + bodies + lists + up(2 * (K + 1))
    if whole <= mid_slab:
        return "warp"
    if whole <= SLAB:
        return "block"
    if bodies + lists + up(16 * K) + RING <= SLAB:
        return "ring"
    return "rows in L2" if bodies + lists + up(2 * (K + 1)) <= SLAB else "rows and bodies in L2"


@pytest.fixture(scope="module")
def pile():
    from rainbow_b200 import scenes
    arrays, _ = scenes.batch_arrays(n_scenes=1, seed=21, pool=3, body_range=(24, 24), resolution=16, device="cuda:0")
    a = {k: (v.cpu().numpy() if hasattr(v, "cpu") else v) for k, v in arrays[0].items() if k != "shape_key"}
    a["body_r"] = np.concatenate([a["body_r"][:1], a["body_r"][1:] * [0.8, 0.7, 0.8]])
    return a


def with_chips(pile, count):
    """The pile's scene with `count` chips and their ground added, 500 m away."""
    if not count:
        return pile
    c, a = chips(count), dict(pile)
    n = len(a["shape_v_off"]) - 1
    for key in ("shape_v_off", "shape_t_off", "shape_g_off"):
        a[key] = np.concatenate([a[key], np.asarray(c[key])[1:] + a[key][-1]])
    c["body_shape"] = c["body_shape"] + n
    c["body_r"] = c["body_r"] + [500.0, 0.0, 0.0]
    for key in ("shape_V", "shape_T", "shape_grid", "shape_grid_meta", "body_shape", "body_r", "body_q", "body_v",
                "body_w", "body_mass", "body_inertia", "body_fixed", "body_material", "body_force_order"):
        a[key] = np.concatenate([np.asarray(a[key]), np.asarray(c[key]).astype(np.asarray(a[key]).dtype)])
    return a


def solve(arrays, scheme, precision="fp32", sweeps=24, **launch):
    """(velocities, impulses, statistics) of one step of a fixed number of sweeps, and the FP64 solver's residual of the
    impulses it returned, from which a step without sweeps started."""
    from rainbow_b200 import world as W
    w = W.DeviceWorld([arrays], device="cuda:0", max_iterations=sweeps)
    x0, u0 = w.state()
    out = None
    for mode, cap in ((precision, sweeps), ("fp64", 0)):
        rp = W.make_rb_params(W.params_from_vector(arrays["params"]), scheme=scheme, termination="residual_fixed_r",
                              residual_tolerance=-1.0, residual_interval=5, precision=mode, warm_start=out is not None)
        rp.max_iterations = cap
        for key, v in launch.items():
            setattr(rp, key, v)
        w.set_state(x0, u0)
        assert w.step(rp) == 0
        if out is None:
            out = w.state()[1], w.contacts()["sol"].reshape(-1, 4), w.stats()[0]
    return out + (w.stats()[0].residual,)


@pytest.mark.parametrize("scheme", ["rigid_gauss_seidel", "parallel_gauss_seidel", "parallel_jacobi"])
def test_size_classes_give_the_same_bits(pile, scheme):
    u0, sol0, st0, res0 = solve(pile, scheme)
    nb, K = len(pile["body_mass"]), len(sol0)
    assert size_class(K, nb) == "warp" and st0.fp32_sweeps == 24 and K > 60 and np.abs(sol0[:, 1:]).max() > 0.0
    np.testing.assert_allclose(st0.residual, res0, rtol=1e-9)   # FP64 sums of ~100 terms in two orders, quotients of 1e4
    small = dict(fp32_small_slab=4096, fp32_mid_slab=8192)
    seen = {"warp"}
    for chip_count, launch in ((0, small), (40, small), (1000, {}), (2750, {}), (3750, {})):
        u, sol, st, res = solve(with_chips(pile, chip_count), scheme, **launch)
        seen.add(size_class(len(sol), nb + chip_count + (chip_count > 0), **({"mid_slab": 8192} if launch else {})))
        assert st.fp32_sweeps == 24 and len(sol) >= K + 0.9 * chip_count
        np.testing.assert_array_equal(sol[:K], sol0)
        np.testing.assert_array_equal(u[:nb], u0)
        np.testing.assert_allclose(st.residual, res, rtol=1e-9)
    assert seen == {"warp", "block", "ring", "rows in L2", "rows and bodies in L2"}

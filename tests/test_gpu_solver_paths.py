"""The solver's launch and team variants against the oracle, FP64, bit for bit.

The block solver takes 256, 128 or 64 threads a scene by the number of scenes, sweeps with one to eight warps by the
width of the levels, and numbers the free bodies that have contacts (with and without a fixed body among the rest);
batches of many scenes go to the warp solver.  Scenes of one body up, and of levels from one contact to wider than
eight warps' quads, at the edges of those rules."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pool():
    """Small piles squeezed together so that their bodies touch from the first step on."""
    from rainbow_b200 import scenes
    arrays, params = scenes.batch_arrays(n_scenes=24, seed=11, pool=3, body_range=(1, 40), resolution=16,
                                         device="cuda:0")
    for a in arrays:
        a["body_r"] = np.concatenate([a["body_r"][:1], a["body_r"][1:] * [0.45, 0.3, 0.45]])
    return arrays, params


def _compare(world, ors, picks, rp, steps, **okw):
    contacts = 0
    for _ in range(steps):
        assert world.step(rp) == 0
        x, u = world.state()
        c = world.contacts()
        st = world.stats()
        for i in picks:
            o = ors[i].step(**okw)
            b0, b1 = world.scene_start[i], world.scene_start[i + 1]
            k0, K = st[i].contact_start, st[i].n_contacts
            assert K == o["n_contacts"]
            contacts += K
            np.testing.assert_array_equal(c["sol"][4 * k0:4 * (k0 + K)], o["sol"])
            if K:
                assert (st[i].iterations, st[i].exitcode) == (o["iterations"], o["exitcode"])
            np.testing.assert_array_equal(x[b0:b1].ravel(), o["x"])
            np.testing.assert_array_equal(u[b0:b1].ravel(), o["u"])
    assert contacts > 0


@pytest.mark.parametrize("scheme,mode", [("rigid_gauss_seidel", 0), ("rigid_gauss_seidel", 2), ("gauss_seidel", 1),
                                         ("parallel_jacobi_hybrid", 0)])
@pytest.mark.parametrize("n_scenes", [1, 148, 149, 297, 4736])
def test_scene_counts(oracle_lib, pool, n_scenes, scheme, mode):
    from rainbow_b200 import world as W
    arrays, params = pool
    many = [arrays[(7 * i) % len(arrays)] for i in range(n_scenes)]
    picks = sorted({0, n_scenes // 2, n_scenes - 1})
    world = W.DeviceWorld(many, device="cuda:0", max_iterations=100)
    rp = W.make_rb_params(params, scheme=scheme, termination=("merit", "residual", "residual_fixed_r")[mode],
                          residual_interval=3)
    rp.max_iterations = 20
    ors = {i: oracle_lib.OracleScene(many[i]) for i in picks}
    for o in ors.values():
        o.set_param("max_iterations", 20)
    _compare(world, ors, picks, rp, 2, scheme=scheme, tol_mode=mode, tol=1e-6, residual_interval=3)


@pytest.mark.parametrize("count,fixed_ground", [(2, True), (40, True), (400, True), (40, False)])
def test_level_widths(oracle_lib, pool, count, fixed_ground):
    """Side-by-side pairs of bodies on one ground: levels of up to `count` contacts; without a fixed body every
    contact's two bodies are free and the ground chains them all."""
    from rainbow_b200 import world as W
    arrays, params = pool
    a = dict(max(arrays, key=lambda s: len(s["body_mass"])))
    n = len(a["body_mass"]) - 1
    side = int(np.ceil(np.sqrt(count)))
    pick = [1 + i % n for i in range(count)]
    for k in ("body_shape", "body_mass", "body_inertia", "body_material", "body_force_order", "body_q", "body_v",
              "body_w", "body_fixed", "body_r"):
        a[k] = np.concatenate([a[k][:1], a[k][pick]])
    place = np.array([[2.6 * (i % side - side / 2), 0.45, 2.6 * (i // side - side / 2)] for i in range(count)])
    a["body_r"] = np.concatenate([a["body_r"][:1], place])
    if not fixed_ground:
        a["body_fixed"] = np.zeros(count + 1, np.uint8)
    world = W.DeviceWorld([a], device="cuda:0", max_iterations=100)
    rp = W.make_rb_params(params)
    o = oracle_lib.OracleScene(a)
    _compare(world, {0: o}, [0], rp, 2)


@pytest.mark.parametrize("slices,resolution", [(4, 12), (8, 12), (16, 12), (24, 10)])
def test_deep_overlaps(oracle_lib, slices, resolution):
    """Spheres of 32 to 1100 triangles deep inside one another and a ground: candidate pairs of one cluster pair up to
    more than the wide mid phase caches, many accepted candidates and duplicates per pair, long contact lists."""
    from rainbow_b200 import api as API, engine_io, geometry as GEO, world as W
    engine = API.create_engine("cuda:0")
    engine.params.resolution = resolution
    engine.params.max_iterations = 5
    API.create_surfaces_interaction(engine, "m", "m", 0.0, np.array([0.4, 0.4, 0.4]))
    V, T = GEO.create_box(8.0, 1.0, 8.0)
    API.create_shape(engine, "ground", API.create_mesh(V, T))
    V, T = GEO.create_sphere(1.5, slices, slices)
    API.create_shape(engine, "ball", API.create_mesh(V, T))
    API.create_gravity_force(engine, "gravity", 9.81, np.array([0.0, 1.0, 0.0]))
    rng = np.random.default_rng(slices)
    for k in range(7):
        name = "b%d" % k
        API.create_rigid_body(engine, name)
        API.connect_shape(engine, name, "ball" if k else "ground")
        API.set_position(engine, name, rng.uniform(-0.7, 0.7, 3) + [0.0, 1.2, 0.0] if k else np.array([0.0, -0.5, 0.0]), True)
        q = rng.normal(size=4)
        API.set_orientation(engine, name, q / np.linalg.norm(q) if k else np.array([1.0, 0.0, 0.0, 0.0]), True)
        API.set_mass_properties(engine, name, 1.0)
        API.set_body_material(engine, name, "m")
        if k:
            API.connect_force(engine, name, "gravity")
        else:
            API.set_body_type(engine, name, "fixed")
    arrays = engine_io.scene_arrays(engine)
    world = W.DeviceWorld([arrays, arrays], device="cuda:0", max_iterations=100)
    o = oracle_lib.OracleScene(arrays)
    rp = W.make_rb_params(W.params_from_vector(arrays["params"]))
    _compare(world, {1: o}, [1], rp, 2, capacity=1 << 15)


@pytest.mark.parametrize("count", [1, 3, 4096, 4097, 16383, 16384, 16385, 40000])
def test_scan_sizes(count):
    """Topology prefix sums (device scans) of as many bodies as one block scans in a round, one more, and of both
    scan variants, against NumPy's."""
    import ctypes
    import torch
    from rainbow_b200 import _native as N
    rng = np.random.default_rng(count)
    nv, nt = rng.integers(4, 400, 5), rng.integers(4, 900, 5)
    shape = rng.integers(0, 5, count).astype(np.int32)
    off = lambda n: torch.from_numpy(np.concatenate([[0], np.cumsum(n)]).astype(np.int32)).cuda()  # noqa: E731
    v_off, t_off, t_shape = off(nv), off(nt), torch.from_numpy(shape).cuda()
    sh, bd = N.RbShapes(), N.RbBodies()
    sh.n_shapes, sh.v_off, sh.t_off = 5, v_off.data_ptr(), t_off.data_ptr()
    sums = [np.concatenate([[0], np.cumsum(n[shape])]) for n in (nv, nt, (nt + 31) // 32)]
    bd.n_bodies, bd.n_scenes, bd.shape = count, 1, t_shape.data_ptr()
    bd.n_body_vertices, bd.n_body_triangles, bd.n_clusters = (int(s[-1]) for s in sums)
    out = [torch.empty(count + 1, dtype=torch.int32, device="cuda") for _ in range(3)]
    owners = [torch.empty(int(s[-1]), dtype=torch.int32, device="cuda") for s in sums]
    for name, t in zip(("body_v0", "body_t0", "body_c0", "vert_body", "tri_body", "clu_body"), out + owners):
        setattr(bd, name, t.data_ptr())
    scratch = torch.empty(N.RB_TOPOLOGY_SCRATCH_BYTES, dtype=torch.uint8, device="cuda")
    N.check(N.load().rb_build_topology(ctypes.byref(sh), ctypes.byref(bd), scratch.data_ptr(), scratch.numel(),
                                       torch.cuda.current_stream().cuda_stream), "rb_build_topology")
    for got, want in zip(out, sums):
        np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("bodies", [700, 1500, 2600])   # rows through the ring, and too many bodies for it
@pytest.mark.parametrize("scheme", ["rigid_gauss_seidel", "parallel_gauss_seidel"])
def test_large_fp32_scenes_match_their_fp64_solve(bodies, scheme):
    """A pile too large for a slab, its rows through the ring or, beyond that, straight from L2: the FP32 solve of a
    step alone in the batch and beside small scenes is the same to the bit, and its impulses give the FP64 residual
    the solver reports (FP32 rounding of a problem with impulses up to 1e4: 1e-3 of the largest velocity)."""
    from rainbow_b200 import scenes, world as W
    big = scenes.batch_arrays(n_scenes=1, seed=3, pool=4, body_range=(bodies, bodies), resolution=16, device="cuda:0",
                              ground=60.0)[0][0]
    small, params = scenes.batch_arrays(n_scenes=3, seed=4, pool=4, body_range=(8, 30), resolution=16, device="cuda:0")
    for a in [big] + small:
        a["body_r"] = np.concatenate([a["body_r"][:1], a["body_r"][1:] * [0.62, 0.5, 0.62]])
    kw = dict(scheme=scheme, termination="residual_fixed_r", residual_interval=4, residual_tolerance=1e-6)
    worlds = [W.DeviceWorld([big], max_iterations=200), W.DeviceWorld(small[:1] + [big] + small[1:], max_iterations=200),
              W.DeviceWorld([big], max_iterations=200)]
    for w, precision in zip(worlds, ("fp32_refine", "fp32_refine", "fp64")):
        rp = W.make_rb_params(params, precision=precision, **kw)
        rp.max_iterations = 200
        assert w.step(rp) == 0
    st = [worlds[0].stats()[0], worlds[1].stats()[1], worlds[2].stats()[0]]
    assert st[0].n_contacts == st[1].n_contacts == st[2].n_contacts > 500
    assert st[0].fp32_sweeps == st[1].fp32_sweeps > 0 and st[0].residual == st[1].residual
    b0, b1 = worlds[1].scene_start[1], worlds[1].scene_start[2]
    u = [worlds[0].state()[1], worlds[1].state()[1][b0:b1], worlds[2].state()[1]]
    np.testing.assert_array_equal(u[0], u[1])
    assert np.max(np.abs(u[0] - u[2])) <= 1e-3 * max(1.0, np.max(np.abs(u[2])))

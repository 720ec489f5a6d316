"""Signed distance grids built on the GPU (grid3.py:320 create_signed_distance, whose igl.signed_distance call
at grid3.py:338 rb_signed_distance_grid replaces) against the grids the reference step consumed in the golden
fixtures, and the batched construction of the per-body workload."""
import numpy as np
import pytest

from conftest import load_fixture

pytestmark = pytest.mark.gpu


def _shapes(d):
    sv, st, sg = (np.asarray(d[k]) for k in ("shape_v_off", "shape_t_off", "shape_g_off"))
    V, T, G = np.asarray(d["shape_V"]).reshape(-1, 3), np.asarray(d["shape_T"]).reshape(-1, 3), np.asarray(d["shape_grid"]).ravel()
    meta = np.asarray(d["shape_grid_meta"]).reshape(-1, 12)
    for k in range(len(sv) - 1):
        yield V[sv[k]:sv[k + 1]], T[st[k]:st[k + 1]], G[sg[k]:sg[k + 1]], meta[k]


def _grid_on_gpu(V, T, meta):
    import ctypes
    import torch
    from rainbow_b200 import _native as N
    tV = torch.from_numpy(np.ascontiguousarray(V, np.float64)).cuda()
    tT = torch.from_numpy(np.ascontiguousarray(T, np.int32)).cuda()
    tM = torch.from_numpy(np.ascontiguousarray(meta, np.float64)).cuda()
    n = int(meta[9] * meta[10] * meta[11])
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    N.check(N.load().rb_signed_distance_grid(tV.data_ptr(), len(V), tT.data_ptr(), len(T), tM.data_ptr(),
                                             out.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
            "rb_signed_distance_grid")
    return out.cpu().numpy()


@pytest.mark.parametrize("name", ["spheres", "c1_boxes64", "boxes8", "tower6"])
def test_gpu_grids_match_the_grids_the_reference_consumed(name):
    """Every shape of the fixture (boxes of several sizes, the ground slab, 16 x 16 spheres): the GPU grid equals
    the grid the reference's own step used, node for node, to 1e-12 (the fixtures' grids came from the NumPy
    restatement of igl.signed_distance: closest point by Ericson's case analysis, sign by the generalized
    winding number)."""
    d = load_fixture(name)
    n = 0
    for V, T, G, meta in _shapes(d):
        got = _grid_on_gpu(V, T, meta)
        np.testing.assert_allclose(got, G, rtol=0.0, atol=1e-12)
        n += 1
    assert n >= 2


def test_batched_grids_equal_single_grids():
    """rb_signed_distance_grids over several meshes equals rb_signed_distance_grid on each, bit for bit."""
    from rainbow_b200 import geometry as GEO
    from rainbow_b200.types import Grid
    meshes = [GEO.create_box(1.0, 0.6, 2.0), GEO.create_sphere(0.7, 16, 16), GEO.create_box(24.0, 1.0, 24.0),
              GEO.create_sphere(0.3, 8, 8)]
    Vs, Ts, metas = [], [], []
    for i, (V, T) in enumerate(meshes):
        V = np.asarray(V, np.float64)
        res = (17, 32, 9, 20)[i]
        metas.append(Grid(V.min(0) - 0.2, V.max(0) + 0.2, res, res + 1, res + 2).meta())
        Vs.append(V)
        Ts.append(np.asarray(T, np.int32))
    values, g_off = GEO.signed_distance_grids(Vs, Ts, metas)
    values = values.cpu().numpy()
    for i in range(len(meshes)):
        np.testing.assert_array_equal(values[g_off[i]:g_off[i + 1]], _grid_on_gpu(Vs[i], Ts[i], metas[i]))


def test_per_body_workload_steps_like_the_oracle(oracle_lib):
    """The batch workload with a shape and grid per body: every body's grid is its own mesh's grid, masses scale
    with size, and the batch steps bit-identically to the oracle on host copies of the same scenes."""
    from rainbow_b200 import scenes, world as W
    arrays, params = scenes.batch_arrays(n_scenes=3, seed=5, pool=None, body_range=(8, 24), resolution=16,
                                         device="cuda:0")
    for a in arrays:
        host = {k: (v.cpu().numpy() if hasattr(v, "cpu") else v) for k, v in a.items()}
        shapes = list(_shapes(host))
        assert len(shapes) == len(a["body_mass"])          # the ground and one shape per body
        for V, T, G, meta in shapes[1:4]:
            np.testing.assert_array_equal(G, _grid_on_gpu(V, T, meta))
        assert len(set(np.round(a["body_mass"][1:], 9))) == len(a["body_mass"]) - 1   # sizes differ per body
    world = W.DeviceWorld(arrays, device="cuda:0", max_iterations=100)
    ors = [oracle_lib.OracleScene({k: (v.cpu().numpy() if hasattr(v, "cpu") else v) for k, v in a.items()})
           for a in arrays]
    rp = W.make_rb_params(params)
    for s in range(8):
        assert world.step(rp) == 0
        x, u = world.state()
        for i, sc in enumerate(ors):
            o = sc.step()
            b0, b1 = world.scene_start[i], world.scene_start[i + 1]
            np.testing.assert_array_equal(x[b0:b1].ravel(), o["x"], err_msg="step %d scene %d" % (s, i))
            np.testing.assert_array_equal(u[b0:b1].ravel(), o["u"], err_msg="step %d scene %d" % (s, i))


def test_per_body_scenes_do_not_depend_on_which_others_are_built():
    """A multi-GPU rank builds only its share of the per-body workload: a selected scene's arrays (shapes,
    grids, bodies) equal the same scene built with all the others, and the counts without building match."""
    from rainbow_b200 import scenes
    every, _ = scenes.batch_arrays_per_body(n_scenes=5, seed=2, body_range=(8, 16), resolution=8, device="cuda:0")
    some, _ = scenes.batch_arrays_per_body(n_scenes=5, seed=2, body_range=(8, 16), resolution=8, device="cuda:0",
                                           select=[1, 4])
    assert [len(a["body_mass"]) for a in every] == scenes.per_body_counts(5, 2, (8, 16))
    for a, b in zip([every[1], every[4]], some):
        for k in a:
            va = a[k].cpu().numpy() if hasattr(a[k], "cpu") else np.asarray(a[k])
            vb = b[k].cpu().numpy() if hasattr(b[k], "cpu") else np.asarray(b[k])
            np.testing.assert_array_equal(va, vb, err_msg=k)


def _plain_grid(V, T, meta):
    """Distance to the nearest triangle and the winding number of every node, summed arc by arc, in NumPy."""
    I, J, K = (int(v) for v in meta[9:12])
    k, j, i = np.meshgrid(np.arange(K), np.arange(J), np.arange(I), indexing="ij")
    P = np.stack([meta[a] + meta[6 + a] * n.ravel() for a, n in zip(range(3), (i, j, k))], axis=1)
    dist, wind = np.full(len(P), np.inf), np.zeros(len(P))
    for tri in V[T]:
        away = [P - c for c in tri]
        n = np.cross(tri[1] - tri[0], tri[2] - tri[0])
        n /= np.linalg.norm(n)
        inside = np.ones(len(P), bool)
        for c in range(3):
            e = tri[(c + 1) % 3] - tri[c]
            t = np.clip(away[c] @ e / (e @ e), 0.0, 1.0)
            dist = np.minimum(dist, np.linalg.norm(away[c] - t[:, None] * e, axis=1))
            inside &= np.cross(e, away[c]) @ n >= 0.0
        dist = np.where(inside, np.minimum(dist, np.abs(away[0] @ n)), dist)
        A, B, C = (-a for a in away)
        la, lb, lc = (np.linalg.norm(a, axis=1) for a in away)
        dots = [(x * y).sum(1) for x, y in ((A, B), (B, C), (C, A))]
        wind += 2.0 * np.arctan2((A * np.cross(B, C)).sum(1), la * lb * lc + dots[0] * lc + dots[1] * la + dots[2] * lb)
    return dist, np.abs(wind) / (4.0 * np.pi)


@pytest.mark.parametrize("mesh,triangles,margin,res", [
    ("box", 12, 0.0, (9, 9, 9)),        # nodes on the corners, edges and faces
    ("box", 12, 0.125, (11, 11, 11)),
    ("box", 10, 0.25, (13, 7, 5)),      # an open box
    ("sphere", 127, 0.1, (7, 32, 3)), ("sphere", 128, 0.1, (33, 4, 4)), ("sphere", 129, 0.1, (5, 5, 31)),
    ("sphere", 448, 0.3, (32, 8, 2)),
    ("nested", 24, 0.2, (17, 17, 17)),  # one box inside another: winding numbers 0, 1 and 2
])
def test_grid_signs_and_distances(mesh, triangles, margin, res):
    """Node for node against the plain evaluation: distances to 1e-12, signs wherever the winding number is not
    within rounding of its threshold; parts of meshes, nodes on the surface and sizes at the edges of the tiles."""
    from rainbow_b200 import geometry as GEO
    from rainbow_b200.types import Grid
    V, T = GEO.create_box(1.0, 1.0, 1.0) if mesh != "sphere" else GEO.create_sphere(0.5, 16, 16)
    V, T = np.asarray(V, np.float64), np.asarray(T, np.int32)
    if mesh == "nested":
        V, T = np.concatenate([V, 0.5 * V]), np.concatenate([T, T + len(V)])
    T = T[:triangles]
    meta = Grid(V.min(0) - margin, V.max(0) + margin, *res).meta()
    got = _grid_on_gpu(V, T, meta)
    dist, wind = _plain_grid(V, T, meta)
    np.testing.assert_allclose(np.abs(got), dist, rtol=0.0, atol=1e-12)
    clear = (np.abs(wind - 0.5) > 1e-9) & (dist > 1e-12)
    assert clear.any()
    np.testing.assert_array_equal((got < 0.0)[clear], (wind > 0.5)[clear])

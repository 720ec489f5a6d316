"""FP64 batches whose scenes differ much in size: the block size goes by the number of scenes, the room that the largest
one's accumulators leave on an SM, and how far it is above the mean; no choice may change a result."""
import numpy as np
import pytest

from test_gpu_fp32_sweeps import chips

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_small,big", [(147, 200), (148, 200), (296, 200), (297, 30), (297, 1200), (297, 2300), (297, 4700)])
def test_a_large_scene_among_small_ones(n_small, big):
    from rainbow_b200 import world as W
    scenes = [chips(1 + i % 9) for i in range(9)]
    many = [scenes[i % 9] for i in range(n_small)]
    many.insert(n_small // 2, chips(big))
    rp = W.make_rb_params(W.params_from_vector(many[0]["params"]))
    worlds = [W.DeviceWorld(many, device="cuda:0"), W.DeviceWorld(scenes, device="cuda:0"), W.DeviceWorld(many[n_small // 2], device="cuda:0")]
    for _ in range(2):
        assert [w.step(rp) for w in worlds] == [0, 0, 0]
    (x, u), (xs, us), (xb, ub) = (w.state() for w in worlds)
    st, s0 = worlds[0].scene_start, worlds[1].scene_start
    assert worlds[0].stats()[n_small // 2].n_contacts > big // 2
    for i in range(n_small + 1):
        if i == n_small // 2:
            wx, wu = xb, ub
        else:
            k = (i - (i > n_small // 2)) % 9
            wx, wu = xs[s0[k]:s0[k + 1]], us[s0[k]:s0[k + 1]]
        np.testing.assert_array_equal(x[st[i]:st[i + 1]], wx)
        np.testing.assert_array_equal(u[st[i]:st[i + 1]], wu)


@pytest.mark.parametrize("n_scenes,bodies", [(297, 63), (297, 66), (1184, 66), (1185, 66)])
def test_even_batches_of_small_and_larger_scenes(n_scenes, bodies):
    from rainbow_b200 import world as W
    one = chips(bodies - 1)
    rp = W.make_rb_params(W.params_from_vector(one["params"]))
    many, alone = W.DeviceWorld([one] * n_scenes, device="cuda:0"), W.DeviceWorld(one, device="cuda:0")
    for _ in range(2):
        assert [w.step(rp) for w in (many, alone)] == [0, 0]
    (x, u), (x1, u1) = many.state(), alone.state()
    assert alone.stats()[0].n_contacts > bodies // 2
    np.testing.assert_array_equal(x.reshape(n_scenes, bodies, 7), np.broadcast_to(x1, (n_scenes, bodies, 7)))
    np.testing.assert_array_equal(u.reshape(n_scenes, bodies, 6), np.broadcast_to(u1, (n_scenes, bodies, 6)))

"""Read-backs of one world from several threads at once."""
import threading

import numpy as np
import pytest

from conftest import load_fixture

pytestmark = pytest.mark.gpu


def test_threads_read_one_world_back_together():
    """Threads that read the contacts, and the state with them, of one stepped world at the same time each get what a
    thread alone gets: the pinned staging is never two calls' at once."""
    import torch
    from rainbow_b200 import world as W
    d = load_fixture("c1_boxes64")
    w = W.DeviceWorld(d)
    for _ in range(3):
        assert w.step(W.make_rb_params(W.params_from_vector(d["params"]))) == 0
    x, u, want = w.state_and_contacts()
    assert len(want["g"]) > 50
    wrong, start = [], threading.Barrier(4)

    def read(with_state):
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait()
            for _ in range(300):
                if with_state:
                    x1, u1, got = w.state_and_contacts()
                    if not (np.array_equal(x, x1) and np.array_equal(u, u1)):
                        wrong.append("state")
                else:
                    got = w.contacts()
                wrong.extend(k for k in want if not np.array_equal(want[k], got[k]))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=read, args=(i % 2 == 0,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

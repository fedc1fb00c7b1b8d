"""Segmentations of several host threads at once, each with a closing ball of its
own: every thread gets the objects that it gets alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volume(seed, shape=(24, 90, 110), n=60):
    """Small blobs, near enough to one another that a larger ball joins more of them."""
    rng = np.random.default_rng(seed)
    v = (1e-3 * rng.random(shape)).astype(np.float32)
    for _ in range(n):
        z, y, x = (int(rng.integers(1, k - 1)) for k in shape)
        v[z - 1:z + 2, y - 1:y + 2, x - 1:x + 2] = 0.3 + 0.7 * rng.random()
    return v


@pytest.mark.parametrize("sizes", [(1, 5), (0, 3, 7, 15)])
def test_threads_with_balls_of_their_own(rihvr, sizes):
    jobs = [(volume(i), rihvr.segment_params(close_size=c, min_intensity=20.0)) for i, c in enumerate(sizes)]
    alone = [rihvr.segment_intensity(v, sp)[0] for v, sp in jobs]
    # the ball matters on these volumes
    assert len({len(rihvr.segment_intensity(jobs[0][0], sp)[0]) for _, sp in jobs}) > 1
    gate = threading.Barrier(len(jobs))
    wrong = []

    def work(i):
        gate.wait()
        for _ in range(25):
            got = rihvr.segment_intensity(*jobs[i])[0]
            if got.tobytes() != alone[i].tobytes():
                wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

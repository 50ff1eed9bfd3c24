"""Several threads read the series of different replicas of one batch at the same time:
each gets its own replica's numbers."""
import threading

import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


def test_series_read_from_several_threads():
    n, sweeps = 8, 40
    reps = [dict(lt=8, lx=4, ly=2 * (i + 2), beta=2.0 + i, boundary=i % 3, hot=1, seed=3 + i) for i in range(n)]
    b = q.Batch(reps, precision="fp32", renorm_every=1)
    b.reserve(sweeps)
    b.init()
    b.run(sweeps, measure_every=1)
    want = [b.series(i, sweeps) for i in range(n)]
    wrong = []
    start = threading.Barrier(n)

    def read(i):
        start.wait()
        for _ in range(300):
            got = b.series(i, sweeps)
            if not all(np.array_equal(g, w) for g, w in zip(got, want[i])):
                wrong.append(i)
                return

    threads = [threading.Thread(target=read, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong

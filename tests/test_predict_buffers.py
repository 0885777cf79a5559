"""Prediction's kept buffers: threads that predict on one network at the same time, with sizes that
make the buffers grow, and a call above the size that is kept, give the bits of calls made alone."""
import threading

import numpy as np
import pytest

from netflux_b200 import surrogate as sur

pytestmark = pytest.mark.gpu


def _features(n, seed):
    return np.random.default_rng(seed).uniform(-1, 1, (n, 7)).astype(np.float32)


def test_threads_on_one_network():
    sizes = (1, 127, 1000, 40000, 129, 150000, 64, 300000)
    feats = [_features(n, k) for k, n in enumerate(sizes)]
    alone = []
    for f in feats:
        alone.append(sur.MLP(3).predict(f)[0])
    m = sur.MLP(3)
    got = [[None] * 4 for _ in feats]

    def work(k):
        for r in range(4):
            got[k][r] = m.predict(feats[k])[0]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(feats))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(feats)):
        for r in range(4):
            assert np.array_equal(got[k][r], alone[k])


def test_more_samples_than_are_kept():
    n = (1 << 22) + 1
    base = _features(4099, 5)
    f = np.tile(base, (-(-n // 4099), 1))[:n]
    m = sur.MLP(4)
    want = m.predict(base)[0]
    got = m.predict(f)[0]
    assert got.shape == (n, 5) and np.array_equal(got[:4099], want) and np.array_equal(got[-1], want[(n - 1) % 4099])

"""List builds in several threads at once, each with its own context and lists
of its own length, all long enough to need more shared memory per block than a
kernel gets unasked: every build succeeds and gives the lists of a build
alone."""
import threading

import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu

ROUNDS = 2000


def cloud(n, edge, seed):
    """n + n sites in a small free box: every site sees most of the others."""
    X = np.empty((2 * n, 4))
    X[:, :3] = edge * np.random.default_rng(seed).random((2 * n, 3))
    X[:, 3] = 0.1
    return X.reshape(-1), n


def test_threads(gpu):
    jobs = [cloud(n, 3.0, n) for n in (490, 320, 470, 330)]  # at most 979, 639, 939 and 659 neighbors
    contexts, want, errors = [], [], []
    try:
        for X, n in jobs:
            g = A.Gpp(n, n)
            contexts.append(g)
            m = g.build_neighbors(X)
            assert 620 < m < 1000
            want.append((m, [g.neighbors(k) for k in range(5)]))

        def work(g, X, m):
            try:
                for _ in range(ROUNDS):
                    assert g.build_neighbors(X) == m
            except Exception as e:
                errors.append(e)

        threads = [threading.Thread(target=work, args=(g, X, w[0])) for g, (X, _), w in zip(contexts, jobs, want)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors
        for g, (m, lists) in zip(contexts, want):
            for k in range(5):
                (oa, ia), (ob, ib) = g.neighbors(k), lists[k]
                assert np.array_equal(oa, ob) and np.array_equal(ia, ib)
    finally:
        for g in contexts:
            g.close()

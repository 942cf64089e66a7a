"""The tick's chunk kernels when a block takes several chunks, of instances
in different states: 1,300 small free clusters give more element and site
chunks than the kernels have blocks (8 per SM, 152 SMs), and they end their
first evaluations, line searches and the hand-over to the FP64 polish at
different ticks.  An instance's results must not depend on how many others
share its launch: the same bits in batches small enough to give every block
at most one chunk."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu

B, SPLIT = 1300, 4


def minimize(inst, Xs, xs, precision):
    with A.Batch(inst, precision=precision) as b:
        b.set_occupancy(np.concatenate(xs))
        X = np.concatenate(Xs)
        b.build_neighbors(X)
        r = b.minimize(X, gatol=1e-4, max_it=25)
        # and again: the counters of the first run's chunks were left at zero
        again = b.minimize(X, gatol=1e-4, max_it=25)
    assert np.array_equal(r.X, again.X) and np.array_equal(r.nfev, again.nfev)
    return r


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_results_do_not_depend_on_the_batch(gpu, precision):
    rng = np.random.default_rng(5)
    inst, Xs, xs = [], [], []
    for k in range(B):
        X, xH, _, box, nPd, nH = A.lattice_fcc((1, 1, 1), periodic=(0, 0, 0), pos_std=0.01 + 0.04 * rng.random(),
                                               sigma=(0.08, 0.12), x_center=0.1 + 0.6 * rng.random(), x_half=0.02,
                                               seed=k)
        inst.append(dict(nPd=nPd, nH=nH, T=250.0 + 300.0 * rng.random(), box=box, periodic=(0, 0, 0)))
        Xs.append(X)
        xs.append(xH)
    whole = minimize(inst, Xs, xs, precision)
    assert np.isfinite(whole.fmin).all() and len(np.unique(whole.nfev)) > 1
    parts = [minimize(inst[i::SPLIT], Xs[i::SPLIT], xs[i::SPLIT], precision) for i in range(SPLIT)]
    n = len(Xs[0])
    for i, p in enumerate(parts):
        assert np.array_equal(p.X.reshape(-1, n), whole.X.reshape(B, n)[i::SPLIT])
        for a in ("fmin", "iters", "nfev", "gnorm", "reason", "mixed_iters", "fp64_iters"):
            assert np.array_equal(getattr(p, a), getattr(whole, a)[i::SPLIT]), (a, i)

"""The minimization of a context without sites (the API takes one): it is at
its minimum at once, with f = 0 and nothing moved, in both drivers' default
and forced forms, as an evaluation of it gives f = 0."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,polish,minimizer,nfev", [("mixed", 0, "default", 1), ("mixed", 1, "default", 2),
                                                             ("mixed", 1, "device", 2), ("fp64", 0, "device", 1)])
def test_empty(gpu, precision, polish, minimizer, nfev):
    X = np.empty(0)
    with A.Gpp(0, 0, precision=precision) as g:
        g.set_minimizer(minimizer)
        assert g.build_neighbors(X) == 0
        f, G = g.eval(X)
        assert f == 0.0 and G.size == 0
        for _ in range(2):  # the second replays the captured tick
            r = g.minimize(X, polish=polish, max_fev=500)
            assert (r.fmin, r.iters, r.nfev, r.gnorm, r.reason) == (0.0, 0, nfev, 0.0, A.CONVERGED_GATOL)
        f, G = g.eval(X)
        assert f == 0.0

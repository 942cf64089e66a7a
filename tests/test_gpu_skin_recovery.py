"""A skin update that fails (more neighbors within rc + skin than a list may
hold) leaves no half-built candidate lists behind: the next update, at
positions the earlier candidates were built at, builds them again and gives
the lists of a full build."""
import numpy as np
import pytest

import a2c_gb300 as A
from a2c_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_update_after_an_overflow(gpu, precision):
    X, xH, _, box, nPd, nH = A.lattice_fcc((5, 5, 6), periodic=(0, 0, 0), pos_std=0.02, sigma=(0.1, 0.1),
                                           x_center=0.2, x_half=0.05, seed=3)
    assert nPd + nH > 1100
    clump = X.reshape(-1, 4).copy()
    clump[:, :3] *= 0.05  # all sites within 2.6 A of one another
    with A.Gpp(nPd, nH, box=box, periodic=(0, 0, 0), precision=precision) as g, \
            A.Gpp(nPd, nH, box=box, periodic=(0, 0, 0)) as ref:
        g.set_neighbor_skin(0.6)
        m, rebuilt = g.update_neighbors(X)
        assert rebuilt
        with pytest.raises(A.A2CError) as e:
            g.update_neighbors(clump.reshape(-1))
        assert e.value.status == N.A2C_ERR_NEIGHBOR_OVERFLOW
        again, rebuilt = g.update_neighbors(X)
        assert rebuilt and again == m
        assert ref.build_neighbors(X) == m
        for k in range(5):
            (oa, ia), (ob, ib) = g.neighbors(k), ref.neighbors(k)
            assert np.array_equal(oa, ob) and np.array_equal(ia, ib)
        assert np.array_equal(g.shell_counts(), ref.shell_counts())

"""Lists count only after their build has succeeded and been checked, in the
coupled loop too: a list update that fails inside it (more neighbors than a
list may hold) leaves a context that refuses evaluations until lists are
built again, and works after that."""
import numpy as np
import pytest

import a2c_gb300 as A
from a2c_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.0, 0.3])
def test_failed_update_in_the_coupled_loop(gpu, skin):
    X, xH, _, box, nPd, nH = A.lattice_fcc((5, 5, 6), periodic=(0, 0, 0), pos_std=0.0, sigma=(0.1, 0.1),
                                           x_center=0.2, x_half=0.05, seed=3)
    dense = X.reshape(-1, 4).copy()
    dense[:, :3] *= 0.28  # a list of its middle sites would hold over 1000 entries
    with A.Gpp(nPd, nH, T=400.0) as g:
        g.set_occupancy(xH)
        g.set_neighbor_skin(skin)
        m, _ = g.update_neighbors(X)
        f0, G0 = g.eval(X)
        with pytest.raises(A.A2CError) as e:  # no iteration: the positions stay
            g.dmd_run(dense.reshape(-1), xH, np.zeros(nH), np.zeros(nH, dtype=np.int32), [], [], 3, dt=1e-30, nu=1e13,
                      Qm=0.23, x_bd=0.8, gamma_bd=2.0, neighbor_update=True, max_it=0)
        assert e.value.status == N.A2C_ERR_NEIGHBOR_OVERFLOW
        with pytest.raises(A.A2CError) as e:
            g.eval(X)
        assert e.value.status == N.A2C_ERR_STATE
        assert g.update_neighbors(X)[0] == m
        g.set_occupancy(xH)
        f1, G1 = g.eval(X)
        assert f1 == f0 and np.array_equal(G1, G0)

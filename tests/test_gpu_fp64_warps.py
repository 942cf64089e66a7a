"""The FP64 passes at the edges of their work split: site counts on either
side of each sites-per-warp choice, a last group that is not full, a warp
that holds the last Pd and the first H sites, empty and uneven lists (free
surfaces, vacancies), zero occupancies, and widths whose quadrature points
reach the exponential tails and leave the fast pair forms' range.  Densities
and gradients equal the oracle's in the device arithmetic bit for bit."""
import numpy as np
import pytest

import a2c_gb300 as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# cells, periodic, sites removed (Pd, H): 512 - 2 sites to 20,480 - 8
CASES = [((4, 4, 4), (1, 1, 1), (1, 1)), ((3, 3, 3), (0, 0, 0), (0, 7)), ((9, 9, 9), (1, 1, 1), (3, 2)),
         ((13, 11, 9), (1, 1, 0), (5, 0)), ((16, 16, 10), (1, 0, 1), (3, 5))]


@pytest.mark.parametrize("cells,periodic,removed", CASES)
def test_passes_equal_the_oracle(gpu, cells, periodic, removed):
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, periodic=periodic, pos_std=0.03, sigma=(0.08, 0.14), x_center=0.3,
                                           x_half=0.2, seed=5)
    rng = np.random.default_rng(1)
    keep = np.ones(nPd + nH, dtype=bool)
    keep[rng.choice(nPd, removed[0], replace=False)] = False
    keep[nPd + rng.choice(nH, removed[1], replace=False)] = False
    X = X.reshape(-1, 4)[keep].copy()
    xH = xH[keep[nPd:]].copy()
    nPd, nH = nPd - removed[0], nH - removed[1]
    X[rng.choice(len(X), 12, replace=False), 3] = 1.2   # points beyond 5.35 A
    X[rng.choice(len(X), 2, replace=False), 3] = 70.0   # points beyond 128 A
    xH[rng.choice(nH, 5, replace=False)] = 0.0
    X = X.reshape(-1)
    pb = O.Problem(nPd, nH, box=box, periodic=periodic)
    off, nbr, *_ = O.neighbors(pb, X)
    with O.arithmetic("device"):
        f_o, G_o, rho_o, _ = O.evaluate(pb, X, xH, off, nbr, mode=1)
    with A.Gpp(nPd, nH, box=box, periodic=periodic) as g:
        g.set_occupancy(xH)
        g.build_neighbors(X)
        f, G = g.eval(X)
        rho = g.density()
    assert np.array_equal(rho, rho_o)
    assert np.array_equal(G, G_o)
    assert f == f_o


def test_an_isolated_site_has_no_neighbors(gpu):
    X = np.array([0.0, 0.0, 0.0, 0.1, 40.0, 0.0, 0.0, 0.1])
    with A.Gpp(1, 1) as g:
        g.set_occupancy(np.array([0.5]))
        assert g.build_neighbors(X) == 0
        _, G = g.eval(X)
    assert np.array_equal(G[:3], np.zeros(3)) and np.array_equal(G[4:7], np.zeros(3))

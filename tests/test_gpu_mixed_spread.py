"""The mixed form's evaluation with more lanes on a site than its sums'
order names (a warp per site for few sites, two lanes in place of one)
against the plain mapping, which an explicit block size selects: the same
bits, for every order, uneven and empty lists, a species boundary inside a
block, and the batched lists."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu

# cells, periodic, sites removed (Pd, H): 1 to 5,825 sites, wide up to 27 per SM
CASES = [((3, 3, 3), (1, 1, 1), (0, 0)), ((4, 3, 5), (0, 0, 0), (3, 1)), ((8, 8, 8), (1, 1, 0), (1, 6)),
         ((9, 9, 9), (1, 1, 1), (2, 5))]


def system(cells, periodic, removed):
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, periodic=periodic, pos_std=0.03, sigma=(0.08, 0.14), x_center=0.3,
                                           x_half=0.2, seed=9)
    rng = np.random.default_rng(2)
    keep = np.ones(nPd + nH, dtype=bool)
    keep[rng.choice(nPd, removed[0], replace=False)] = False
    keep[nPd + rng.choice(nH, removed[1], replace=False)] = False
    X = X.reshape(-1, 4)[keep].copy()
    X[rng.choice(len(X), 9, replace=False), 3] = 0.9  # points beyond the switch radius
    return X.reshape(-1), xH[keep[nPd:]].copy(), box, nPd - removed[0], nH - removed[1]


@pytest.mark.parametrize("cells,periodic,removed", CASES)
@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
def test_same_bits(gpu, cells, periodic, removed, lanes):
    X, xH, box, nPd, nH = system(cells, periodic, removed)
    with A.Gpp(nPd, nH, box=box, periodic=periodic, precision="mixed") as g:
        g.set_occupancy(xH)
        g.build_neighbors(X)
        g.set_tile(lanes, 256, 256)
        f0, G0 = g.eval(X)
        g.set_tile(lanes, 0, 0)
        f1, G1 = g.eval(X)
    assert f1 == f0
    assert np.array_equal(G1, G0)


@pytest.mark.parametrize("lanes", [1, 4])
def test_same_bits_in_a_batch(gpu, lanes):
    inst, Xs, xs = [], [], []
    for k, (cells, periodic, removed) in enumerate(CASES[:2]):
        X, xH, box, nPd, nH = system(cells, periodic, removed)
        inst.append(dict(nPd=nPd, nH=nH, T=250.0 + 100 * k, box=box, periodic=periodic))
        Xs.append(X)
        xs.append(xH)
    X = np.concatenate(Xs)
    with A.Batch(inst, precision="mixed") as b:
        b.set_occupancy(np.concatenate(xs))
        b.build_neighbors(X)
        b.set_tile(lanes, 256, 256)
        f0, G0 = b.eval(X)
        b.set_tile(lanes, 0, 0)
        f1, G1 = b.eval(X)
    assert np.array_equal(f1, f0) and np.array_equal(G1, G0)


def test_a_single_site(gpu):
    X = np.array([1.0, 2.0, 3.0, 0.1])
    with A.Gpp(1, 0, precision="mixed") as g:
        assert g.build_neighbors(X) == 0
        f, G = g.eval(X)
        g.set_tile(4, 256, 256)
        f0, G0 = g.eval(X)
    assert f == f0 and np.array_equal(G, G0)

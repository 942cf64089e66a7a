"""Pass 2 of the mixed form with eight copies of f_Pd' (that table ending at
5.8 A) against the shape with one copy of the whole table, which a block of
512 threads selects: the same bits at the smallest sizes that take the
copies, with points far beyond the shorter table's end, uneven lists, a
remainder of sites, and in a batch's work list."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu

# threads per site, cells: 121,600 / threads sites or a little more, 152 SMs
CASES = [(8, (13, 13, 12), (1, 1, 0), (1, 6)), (4, (16, 16, 15), (0, 0, 0), (3, 1)),
         (2, (20, 20, 20), (1, 1, 1), (11, 30)), (1, (25, 25, 25), (1, 1, 1), (2, 5))]


def system(cells, periodic, removed):
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, periodic=periodic, pos_std=0.03, sigma=(0.08, 0.14), x_center=0.3,
                                           x_half=0.2, seed=9)
    rng = np.random.default_rng(2)
    keep = np.ones(nPd + nH, dtype=bool)
    keep[rng.choice(nPd, removed[0], replace=False)] = False
    keep[nPd + rng.choice(nH, removed[1], replace=False)] = False
    X = X.reshape(-1, 4)[keep].copy()
    X[rng.choice(len(X), 400, replace=False), 3] = 0.9  # points out to 7.5 A
    return X.reshape(-1), xH[keep[nPd:]].copy(), box, nPd - removed[0], nH - removed[1]


@pytest.mark.parametrize("lanes,cells,periodic,removed", CASES)
def test_same_bits(gpu, lanes, cells, periodic, removed):
    X, xH, box, nPd, nH = system(cells, periodic, removed)
    with A.Gpp(nPd, nH, box=box, periodic=periodic, precision="mixed") as g:
        g.set_occupancy(xH)
        g.build_neighbors(X)
        g.set_tile(lanes, 256, 512)
        f0, G0 = g.eval(X)
        for blocks in ((256, 256), (0, 0)):
            g.set_tile(lanes, *blocks)
            f1, G1 = g.eval(X)
            assert f1 == f0 and np.array_equal(G1, G0)


def test_same_bits_in_a_batch(gpu):
    inst, Xs, xs = [], [], []
    for k, (_, cells, periodic, removed) in enumerate(CASES[:2]):
        X, xH, box, nPd, nH = system(cells, periodic, removed)
        inst.append(dict(nPd=nPd, nH=nH, T=250.0 + 100 * k, box=box, periodic=periodic))
        Xs.append(X)
        xs.append(xH)
    X = np.concatenate(Xs)
    with A.Batch(inst, precision="mixed") as b:
        b.set_occupancy(np.concatenate(xs))
        b.build_neighbors(X)
        b.set_tile(4, 256, 512)
        f0, G0 = b.eval(X)
        b.set_tile(4, 256, 256)
        f1, G1 = b.eval(X)
    assert np.array_equal(f1, f0) and np.array_equal(G1, G0)

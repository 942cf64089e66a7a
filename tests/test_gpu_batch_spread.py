"""A batch's work lists under the mappings with more lanes on a site than its
sums' order names (tile.h): a warp for a site while there are few, two lanes
in place of one, the latter with and without the copies of pass 2's tables --
evaluation and minimization have the bits of the plain mapping, which a
pass-2 block of 512 threads selects; so has the tile that is read back."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu

# lanes, cells of the instances: 408, 1,080 and 504 sites (a warp each), 9,576 (two lanes), 66,792 (and table copies)
CASES = [(4, [(3, 3, 3), (4, 2, 3)]), (8, [(4, 3, 5), (3, 5, 5)]), (1, [(3, 3, 4), (3, 3, 3)]),
         (1, [(9, 9, 9), (9, 7, 7), (3, 3, 3)]), (1, [(18, 20, 21), (9, 9, 9), (3, 4, 5)])]


def batch(cells):
    inst, Xs, xs = [], [], []
    for k, c in enumerate(cells):
        per = (1, 1, 0) if k % 2 == 0 else (0, 0, 0)
        X, xH, _, box, nPd, nH = A.lattice_fcc(c, periodic=per, pos_std=0.03, sigma=(0.08, 0.14), x_center=0.3,
                                               x_half=0.2, seed=9 + k)
        X = X.reshape(-1, 4).copy()
        X[3, 3] = 0.9  # points beyond the switch radius
        inst.append(dict(nPd=nPd, nH=nH, T=250.0 + 100 * k, box=box, periodic=per))
        Xs.append(X.reshape(-1))
        xs.append(xH)
    return inst, np.concatenate(Xs), np.concatenate(xs)


@pytest.mark.parametrize("lanes,cells", CASES)
def test_same_bits(gpu, lanes, cells):
    inst, X, xH = batch(cells)
    out = []
    with A.Batch(inst, precision="mixed") as b:
        b.set_occupancy(xH)
        b.build_neighbors(X)
        plain = (lanes, 256, 512)
        b.set_tile(lanes, 0, 0)
        again = b.tile()
        for tile in (plain, (lanes, 0, 0), again):
            b.set_tile(*tile)
            f, G = b.eval(X)
            r = b.minimize(X, polish=0, max_it=6, gatol=1e-9)
            out.append((f, G, r.X, r.fmin, r.nfev))
    for o in out[1:]:
        for a, c in zip(out[0], o):
            assert np.array_equal(a, c)

"""The mixed form's chemical potential, several lanes to an H site, where
the lists do not fill the lanes: one H site (no H neighbors), few, blocks
with a remainder, free surfaces.  Against the FP64 form, with the bound of
the mixed form's other test of it."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu


# H sites kept: one, a few (sparse lists), a block of 256 threads and some, all
@pytest.mark.parametrize("cells,keep", [((3, 3, 3), 1), ((4, 3, 3), 7), ((4, 4, 5), 67), ((7, 5, 6), 837)])
def test_follows_fp64(gpu, cells, keep):
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, periodic=(0, 1, 0), pos_std=0.02, sigma=(0.08, 0.12), x_center=0.4,
                                           x_half=0.2, seed=11)
    rng = np.random.default_rng(3)
    h = np.sort(rng.choice(nH, keep, replace=False))
    X = np.concatenate([X[:4 * nPd], X.reshape(-1, 4)[nPd + h].reshape(-1)])
    full = (rng.random(keep) < 0.1).astype(np.int32)
    full[0] = 0
    out = {}
    for precision in ("fp64", "mixed"):
        with A.Gpp(nPd, keep, box=box, periodic=(0, 1, 0), precision=precision) as g:
            g.set_occupancy(xH[h])
            g.build_neighbors(X)
            out[precision] = g.chem_potential(2.5, np.zeros(keep), full)
    assert np.array_equal(out["mixed"][1], out["fp64"][1])
    assert np.abs(out["mixed"][0] - out["fp64"][0]).max() < 1e-4

"""The cell-list build and the skin re-filter where their grid and their
warps can go wrong: periodic directions of one, two and many cells, sites
outside the box (the entry points take [-L/2, 3L/2]) and on its faces, free
directions with one site's extent, more candidates than a warp's queue, long
lists, and a site count that is no multiple of a block's.  Lists, shell
counts and first H shells equal the oracle's."""
import numpy as np
import pytest

import a2c_gb300 as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu
a0 = 3.89


def lattice(cells, periodic, seed):
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, periodic=periodic, pos_std=0.05, seed=seed)
    return X.reshape(-1, 4).copy(), box, nPd, nH


def outside(cells, periodic, seed):
    """Every site in any of its images within [-L/2, 3L/2], some on a face."""
    X, box, nPd, nH = lattice(cells, periodic, seed)
    rng = np.random.default_rng(seed)
    for d in range(3):
        if periodic[d]:
            L = box[d]
            q = X[:, d] % L + L * rng.integers(-1, 2, len(X))
            X[:, d] = np.where((q < -0.5 * L) | (q > 1.5 * L), X[:, d] % L, q)
            X[:8, d] = [0.0, -0.0, L, np.nextafter(L, 0), np.nextafter(L, 2 * L), -0.5 * L, 1.5 * L, 1e-9]
    return X, box, nPd, nH


def gas(n, edge, seed):
    rng = np.random.default_rng(seed)
    X = np.empty((2 * n, 4))
    X[:, :3] = edge * rng.random((2 * n, 3))
    X[:, 3] = 0.1
    return X, (0.0, 0.0, 0.0), n, n


CASES = {
    "two_cells": (lattice, (3, 3, 3), (1, 1, 1)),
    "two_and_many": (lattice, (4, 3, 9), (1, 1, 1)),
    "slab": (lattice, (5, 7, 4), (1, 0, 1)),
    "outside_two": (outside, (4, 4, 4), (1, 1, 1)),
    "outside_many": (outside, (7, 6, 8), (1, 1, 0)),
    "free": (lattice, (3, 5, 4), (0, 0, 0)),
    "gas": (gas, 331, 11.0),
    "sheet": (gas, 100, np.array([30.0, 20.0, 0.0])),
    "sparse": (gas, 400, np.array([200.0, 150.0, 180.0])),
    "pair": (gas, 1, 3.0),
}


@pytest.mark.parametrize("case", list(CASES))
def test_lists_equal_the_oracle(gpu, case):
    make, shape, spec = CASES[case]
    if make is gas:
        X, box, nPd, nH = gas(shape, spec, 3)
        periodic = (0, 0, 0)
    else:
        periodic = spec
        X, box, nPd, nH = make(shape, periodic, 3)
    X = X.reshape(-1)
    pb = O.Problem(nPd, nH, box=box, periodic=periodic)
    off, nbr, shell, off1, hh1 = O.neighbors(pb, X)
    want = O.split_lists(nPd, nH, off, nbr)
    with A.Gpp(nPd, nH, box=box, periodic=periodic) as g:
        roomy = all(not p or L > 2 * (5.35 + 0.5) for p, L in zip(periodic, box))
        for build in ("cells", "skin") if roomy else ("cells",):
            if build == "skin":
                g.set_neighbor_skin(0.5)
                most, _ = g.update_neighbors(X)
            else:
                most = g.build_neighbors(X)
            assert most == int(np.diff(off).max())
            for lid, name in enumerate(("PdPd", "PdH", "HPd", "HH")):
                go, gi = g.neighbors(lid)
                assert np.array_equal(go, want[name][0]) and np.array_equal(gi, want[name][1]), (build, name)
            go, gi = g.neighbors(4)
            assert np.array_equal(go, off1) and np.array_equal(gi, hh1), build
            assert np.array_equal(g.shell_counts(), shell), build


def test_too_many_neighbors_is_an_error(gpu):
    X, _, nPd, nH = gas(900, 4.0, 1)
    with A.Gpp(nPd, nH) as g:
        with pytest.raises(A.A2CError):
            g.build_neighbors(X.reshape(-1))
        far = X.copy()
        far[:, :3] *= 10.0
        assert g.build_neighbors(far.reshape(-1)) < 1000  # the context stays usable

"""The list builds' scratch and the second pass that lists longer than it
take.

Lists: a few sites in a dense clump make lists several times the others'
length (written in place by a second pass at every build), all sites dense
(the first build takes the second pass, later ones the longer stride), the
same again in the skin path; against the oracle, twice from each context.

Memory held after a build: one dense clump in a large system, or a sparse
gas whose cell grid far outnumbers its sites, must not leave scratch in
proportion to the longest list or to the grid.  The bound is 2,000 bytes a
site: the context's own arrays take about 160 (positions, gradient,
occupancy, densities, partial sums, offsets, shells), the lists of 80 to 90
entries 340 to 360 with the first H shells, the scratch 90 to 130 and at most
512 (128 entries) for the unpacked lists, 1,200 in all, and allocations are
rounded up to 2 MiB; a stride as long as the clump's lists alone would take
3,500, the grid of the gas 400,000."""
import numpy as np
import pytest

import a2c_gb300 as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def with_clump(cells, inside, seed):
    """A periodic lattice with `inside` of its H sites moved into a ball of
    2 A radius around one place."""
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, periodic=(1, 1, 1), pos_std=0.03, seed=seed)
    X = X.reshape(-1, 4).copy()
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(inside, 3))
    u *= (2.0 * rng.random(inside) ** (1 / 3) / np.linalg.norm(u, axis=1))[:, None]
    X[nPd + rng.choice(nH, inside, replace=False), :3] = 0.4 * np.array(box) + u
    return X.reshape(-1), box, (1, 1, 1), nPd, nH


def cloud(n, edge, seed):
    X = np.empty((2 * n, 4))
    X[:, :3] = edge * np.random.default_rng(seed).random((2 * n, 3))
    X[:, 3] = 0.1
    return X.reshape(-1), (0.0, 0.0, 0.0), (0, 0, 0), n, n


CASES = {"clump": lambda: with_clump((9, 8, 8), 500, 5), "short_clump": lambda: with_clump((6, 6, 6), 97, 7),
         "dense": lambda: cloud(400, 7.0, 3)}


@pytest.mark.parametrize("case", list(CASES))
def test_long_lists_equal_the_oracle(gpu, case):
    X, box, periodic, nPd, nH = CASES[case]()
    pb = O.Problem(nPd, nH, box=box, periodic=periodic)
    off, nbr, shell, off1, hh1 = O.neighbors(pb, X)
    want = O.split_lists(nPd, nH, off, nbr)
    with A.Gpp(nPd, nH, box=box, periodic=periodic) as g:
        for build in ("cells", "cells", "skin", "skin"):
            if build == "skin":
                g.set_neighbor_skin(0.1)  # drops the candidate lists: each update builds them
                most, rebuilt = g.update_neighbors(X)
                assert rebuilt
            else:
                most = g.build_neighbors(X)
            assert most == int(np.diff(off).max()) > 128
            for lid, name in enumerate(("PdPd", "PdH", "HPd", "HH")):
                go, gi = g.neighbors(lid)
                assert np.array_equal(go, want[name][0]) and np.array_equal(gi, want[name][1]), (build, name)
            go, gi = g.neighbors(4)
            assert np.array_equal(go, off1) and np.array_equal(gi, hh1), build
            assert np.array_equal(g.shell_counts(), shell), build


@pytest.mark.parametrize("case", ["clump", "gas"])
def test_memory_held(gpu, case):
    import torch

    X, box, periodic, nPd, nH = (with_clump((28, 28, 28), 850, 5) if case == "clump" else cloud(10_000, 2600.0, 1))
    with A.Gpp(4, 4) as g:  # the library is loaded
        g.build_neighbors(cloud(4, 5.0, 1)[0])
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with A.Gpp(nPd, nH, box=box, periodic=periodic) as g:
        m = g.build_neighbors(X)
        assert (900 < m <= 1000) if case == "clump" else m < 10
        held = before - torch.cuda.mem_get_info()[0]
        assert held < 2000 * (nPd + nH) + (64 << 20), held / (nPd + nH)

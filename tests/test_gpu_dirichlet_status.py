"""The Dirichlet condition when the context still holds a flag of an earlier
asynchronous evaluation: the call reports it, and the condition is applied in
the caller's arrays as in the context."""
import ctypes as C

import numpy as np
import pytest

import a2c_gb300 as A
from a2c_gb300 import _native as N

pytestmark = pytest.mark.gpu


def test_applied_with_a_pending_flag(gpu):
    import torch

    X, xH, surf, box, nPd, nH = A.lattice_fcc(3, periodic=(1, 1, 1), pos_std=0.02, sigma=(0.1, 0.1), x_center=0.3,
                                              x_half=0.1, seed=2)
    sites = np.array([1, 5, 7], dtype=np.int32)
    with A.Gpp(nPd, nH, box=box, periodic=(1, 1, 1)) as g:
        g.set_occupancy(xH)
        g.build_neighbors(X)
        bad = X.copy()
        bad[4 * 3] = np.nan
        dX = torch.from_numpy(bad).cuda()
        df, dG = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(dX)
        g.eval_device(dX.data_ptr(), df.data_ptr(), dG.data_ptr())
        for want in (N.A2C_ERR_NONFINITE, N.A2C_OK):
            gamma, full = np.zeros(nH), np.zeros(nH, dtype=np.int32)
            s = N.lib().a2c_gpp_apply_dirichlet(g.handle, N.ptr(sites), C.c_int(3), C.c_double(2.5), C.c_double(0.8),
                                                N.ptr(gamma), N.ptr(full))
            assert s == want
            flag = np.isin(np.arange(nH), sites)
            assert np.array_equal(gamma, np.where(flag, 2.5, 0.0)) and np.array_equal(full, flag.astype(np.int32))
        assert np.array_equal(g.occupancy()[sites], np.full(3, 0.8))

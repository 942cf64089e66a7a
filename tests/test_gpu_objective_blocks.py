"""The mixed form's objective summed by the first blocks of the kernel that
completes the gradient, against its own launch (which the stage timing
keeps): the same bits from one block to the largest grid, and the context's
state is the one evaluated."""
import numpy as np
import pytest

import a2c_gb300 as A

pytestmark = pytest.mark.gpu


# sites: within one block of 256, a few blocks, 2 blocks on each of 152 SMs (77,824 sites) and a remainder
@pytest.mark.parametrize("cells", [(3, 3, 3), (5, 5, 4), (21, 21, 21), (22, 22, 21)])
def test_same_bits(gpu, cells):
    torch = pytest.importorskip("torch")
    X, xH, _, box, nPd, nH = A.lattice_fcc(cells, pos_std=0.03, sigma=(0.08, 0.14), x_center=0.3, x_half=0.2, seed=4)
    with A.Gpp(nPd, nH, box=box, precision="mixed") as g:
        g.set_occupancy(xH)
        g.build_neighbors(X)
        room = torch.zeros(4 * (nPd + nH) + 1, dtype=torch.float64, device="cuda")
        dX = room[1:]  # 8-byte alignment is enough
        dX.copy_(torch.from_numpy(X))
        out = [(torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(dX)) for _ in range(2)]
        torch.cuda.synchronize()
        g.profile_eval(dX.data_ptr(), out[0][0].data_ptr(), out[0][1].data_ptr())
        g.eval_device(dX.data_ptr(), out[1][0].data_ptr(), out[1][1].data_ptr())
        assert np.array_equal(g.state(), X)
        torch.cuda.synchronize()
        f, G = g.eval(X)
    assert out[0][0].item() == out[1][0].item() == f
    assert torch.equal(out[0][1], out[1][1])
    assert np.array_equal(out[1][1].cpu().numpy(), G)

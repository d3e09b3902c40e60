"""Calls at each side of the small-tensor kernel's rule: many tiles over a short
contraction, and ranks that leave most of a tile empty.  Small integers, exact
in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R", [((2, 6, 5000), 64), ((9, 5, 2291), 33), ((12, 18, 932), 34), ((996, 2), 41),
                                    ((947, 2), 40), ((10, 1000, 1000), 1), ((50, 60, 60), 9), ((3, 2, 1500), 8)])
def test_each_side_of_the_rule(cd, dev, dims, R):
    import torch
    rng = np.random.default_rng(sum(dims) + R)
    X = rng.integers(-2, 3, int(np.prod(dims))).astype(np.float64)
    U = [rng.integers(-1, 2, (R, d)).astype(np.float64) for d in dims]
    dX = torch.from_numpy(X).float().cuda()
    dU = [torch.from_numpy(u.reshape(-1)).float().cuda() for u in U]
    for mode in range(len(dims)):
        T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
        kr = np.ones((1, R))
        for m, u in enumerate(U):
            if m != mode:
                kr = (u.T[:, None, :] * kr[None, :, :]).reshape(-1, R)
        for prec in (cd.PREC_FP32, cd.PREC_DEFAULT):
            out = torch.full((dims[mode] * R,), 7.0, device="cuda")
            cd.mttkrp(dX, dims, dU, mode, R, out, prec)
            assert np.array_equal(out.cpu().numpy().reshape(dims[mode], R, order="F").astype(np.float64), T @ kr), mode

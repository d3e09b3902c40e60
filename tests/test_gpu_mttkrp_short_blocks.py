"""MTTKRP where the fastest factor has few rows (2 to 31): the flat-step kernel
or the one that walks row blocks, at each side of the rule between them, in
FP32 and with rounded operands, past the small-tensor kernel.  Small integers,
exact in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R", [((2, 300, 301), 64), ((3, 5, 301, 41), 64), ((3, 301, 301), 20), ((5, 6, 3001), 33),
                                    ((7, 9, 11, 13, 15), 12), ((13, 301, 101), 64), ((17, 301, 101), 64),
                                    ((31, 301, 65), 30), ((301, 2, 301), 64), ((301, 24, 101), 65)])
@pytest.mark.parametrize("prec", ["fp32", "fp16", "bf16", "default"])
def test_short_blocks(cd, dev, dims, R, prec):
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
        out = torch.full((dims[mode] * R,), 7.0, device="cuda")
        cd.mttkrp(dX, dims, dU, mode, R, out, cd.PRECISIONS[prec])
        assert np.array_equal(out.cpu().numpy().reshape(dims[mode], R, order="F").astype(np.float64), T @ kr), mode

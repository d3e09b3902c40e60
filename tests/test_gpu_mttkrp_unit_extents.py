"""MTTKRP over modes of extent 1 in every place (a squeezed tensor's data with
the unit modes kept): such a mode must neither become the factor whose row
blocks the kernels walk nor lose its factor's row.  Sizes past the small-tensor
kernel, against FP64 on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 150, 170), (150, 1, 170), (150, 170, 1), (1, 1, 130, 190), (1, 130, 1, 190),
                                  (60, 1, 50, 1, 9), (1, 25000, 1), (25000, 1, 1)])
@pytest.mark.parametrize("prec,R", [("fp32", 20), ("fp32", 33), ("fp16", 20), ("f64", 20)])
def test_unit_extents(cd, dev, dims, prec, R):
    import torch
    rng = np.random.default_rng(sum(dims) + R)
    # small integers: products and sums exact in every precision (|sum| < 2^24)
    X = rng.integers(-2, 3, int(np.prod(dims))).astype(np.float64)
    U = [rng.integers(-2, 3, (R, d)).astype(np.float64) for d in dims]
    dtype = torch.float64 if prec == "f64" else torch.float32
    dX = torch.from_numpy(X).to(dtype).cuda()
    dU = [torch.from_numpy(u.reshape(-1)).to(dtype).cuda() for u in U]
    for mode in range(len(dims)):
        T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
        kr = np.ones((1, R))
        for m, u in enumerate(U):
            if m != mode:
                kr = (u.T[:, None, :] * kr[None, :, :]).reshape(-1, R)
        want = T @ kr
        out = torch.full((dims[mode] * R,), 7.0, device="cuda", dtype=dtype)
        if prec == "f64":
            cd.mttkrp_f64(dX, dims, dU, mode, R, out)
        else:
            cd.mttkrp(dX, dims, dU, mode, R, out, cd.PRECISIONS[prec])
        assert np.array_equal(out.cpu().numpy().reshape(dims[mode], R, order="F").astype(np.float64), want), mode

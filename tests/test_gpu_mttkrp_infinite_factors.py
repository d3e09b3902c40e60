"""MTTKRP with an infinite factor entry, in each factor in turn, over extents
that end a row block of the fastest factor in every remainder: with positive
data the entry's rank column is +infinity in every row, and the other columns
are those without it.  Nothing past a block's end may turn it into NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(X, dims, U, mode):
    T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
    kr = None
    for m, u in enumerate(U):
        if m != mode:
            kr = u.T if kr is None else (u.T[:, None, :] * kr[None, :, :]).reshape(-1, u.shape[0])
    return T @ kr


@pytest.mark.parametrize("dims,R", [((17, 18, 19), 5), ((34, 35, 33), 20), ((21, 9, 6, 5), 9), ((150, 131, 40), 33)])
@pytest.mark.parametrize("prec", ["f64", "fp32"])
def test_infinite_factor_entry(cd, dev, dims, R, prec):
    import torch
    rng = np.random.default_rng(sum(dims) + R)
    dtype = np.float64 if prec == "f64" else np.float32
    X = rng.random(int(np.prod(dims))).astype(dtype) + 0.5
    U = [rng.random((R, d)).astype(dtype) + 0.5 for d in dims]
    dX = torch.from_numpy(X).cuda()
    for mode in range(len(dims)):
        want = _want(X.astype(np.float64), dims, [u.astype(np.float64) for u in U], mode)
        for f in range(len(dims)):
            if f == mode:
                continue
            V = [u.copy() for u in U]
            V[f][R - 1, dims[f] - 1] = np.inf
            dU = [torch.from_numpy(v.reshape(-1)).cuda() for v in V]
            out = torch.empty(dims[mode] * R, device="cuda", dtype=dX.dtype)
            if prec == "f64":
                cd.mttkrp_f64(dX, dims, dU, mode, R, out)
            else:
                cd.mttkrp(dX, dims, dU, mode, R, out, cd.PREC_FP32)
            got = out.cpu().numpy().reshape(dims[mode], R, order="F")
            assert np.all(np.isposinf(got[:, R - 1])), (mode, f)
            # positive terms: no cancellation, so the sum's own relative error
            eps = 2.0 ** -53 if prec == "f64" else 2.0 ** -24
            assert np.all(np.abs(got[:, : R - 1] - want[:, : R - 1]) <= 64 * eps * want[:, : R - 1])

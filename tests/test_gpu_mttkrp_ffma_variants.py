"""The FP32 FFMA MTTKRP's variants -- 1, 2, 4 and 8 rank lanes of 4 to 8 ranks,
16- and 4-byte copies, rows around 128, blocks that end in every remainder of a
stage, 2nd- to 6th-order tensors -- at sizes that the dispatcher gives to it:
past the small-tensor kernel, and with blocks too long for the flat-step one.
Small integers, exact in FP32; and infinities beside a ragged block's end."""
import os
import re

import numpy as np
import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu


def _assert_route(dims, mode, R):
    """Neither the small-tensor kernel nor the flat-step one takes the call,
    by the limits in the sources."""
    small = open(os.path.join(PKG, "csrc", "mttkrp_small.cu")).read()
    rank, work, K = re.search(r"return R <= (\d+) && work <= (\S+) && K <= (\S+) &&", small).groups()
    n = int(np.prod(dims))
    assert R > int(rank) or n * R > float(work) or n // dims[mode] > float(K)
    rows = re.search(r"return rows0 < (\d+) &&", open(os.path.join(PKG, "csrc", "mttkrp.cu")).read()).group(1)
    assert next(d for m, d in enumerate(dims) if m != mode and d > 1) >= int(rows)


def _khatri_rao(U, mode):
    kr = np.ones((1, U[0].shape[0]))
    for m, u in enumerate(U):
        if m != mode:
            kr = (u.T[:, None, :] * kr[None, :, :]).reshape(-1, u.shape[0])
    return kr


CASES = ([((128, 160, 180), R) for R in (3, 5, 6, 7, 8)] + [((129, 161, 181), R) for R in (3, 5, 6, 7, 8)]
         + [((127, 96, 132), R) for R in (9, 12, 14, 16)] + [((132, 97, 129), R) for R in (9, 12, 14, 16)]
         + [((36, 257, 133), R) for R in (17, 24, 28, 32)] + [((35, 255, 130), R) for R in (17, 28)]
         + [((64, 33, 34, 20), 20), ((33, 32, 3, 5, 7, 9), 20), ((2500, 300), 20), ((301, 2803), 13),
            ((100, 98, 101), 40), ((100, 99, 97), 56), ((44, 63, 65), 150)])


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dims,R", CASES)
def test_variants(cd, dev, dims, R, offset):
    import torch
    rng = np.random.default_rng(sum(dims) + R)
    X = rng.integers(-2, 3, int(np.prod(dims))).astype(np.float64)
    U = [rng.integers(-1, 2, (R, d)).astype(np.float64) for d in dims]
    buf = torch.empty(X.size + 4, device="cuda")
    dX = buf[offset: offset + X.size]
    dX.copy_(torch.from_numpy(X))
    dU = [torch.from_numpy(u.reshape(-1)).float().cuda() for u in U]
    for mode in range(len(dims)):
        _assert_route(dims, mode, R)
        T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
        out = torch.full((dims[mode] * R,), 7.0, device="cuda")
        cd.mttkrp(dX, dims, dU, mode, R, out, cd.PREC_FP32)
        got = out.cpu().numpy().reshape(dims[mode], R, order="F").astype(np.float64)
        assert np.array_equal(got, T @ _khatri_rao(U, mode)), mode


@pytest.mark.parametrize("dims,R", [((130, 131, 133), 6), ((132, 131, 130), 6), ((38, 197, 135), 20), ((35, 99, 134), 30)])
def test_infinities(cd, dev, dims, R):
    """An infinity in X, in the last kappas of a block, makes its own row of M
    infinite and no other; one in a factor its own rank column."""
    import torch
    rng = np.random.default_rng(R)
    X = (rng.random(int(np.prod(dims))) + 0.5).astype(np.float32)
    U = [(rng.random((R, d)) + 0.5).astype(np.float32) for d in dims]
    at = (dims[0] - 1, dims[1] - 1, dims[2] // 2)
    Y = X.copy()
    Y[at[0] + dims[0] * (at[1] + dims[1] * at[2])] = np.inf
    dX, dY = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda()
    for mode in range(3):
        _assert_route(dims, mode, R)
        out = torch.empty(dims[mode] * R, device="cuda")
        cd.mttkrp(dY, dims, [torch.from_numpy(u.reshape(-1)).cuda() for u in U], mode, R, out, cd.PREC_FP32)
        got = out.cpu().numpy().reshape(dims[mode], R, order="F")
        assert np.all(np.isposinf(got[at[mode]])) and np.all(np.isfinite(np.delete(got, at[mode], axis=0)))
        for f in range(3):
            if f == mode:
                continue
            V = [u.copy() for u in U]
            V[f][R - 1, dims[f] - 1] = np.inf
            cd.mttkrp(dX, dims, [torch.from_numpy(v.reshape(-1)).cuda() for v in V], mode, R, out, cd.PREC_FP32)
            got = out.cpu().numpy().reshape(dims[mode], R, order="F")
            assert np.all(np.isposinf(got[:, R - 1])) and np.all(np.isfinite(got[:, : R - 1])), (mode, f)

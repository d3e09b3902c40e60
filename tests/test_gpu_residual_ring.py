"""The tensor-core CP residual (residual_tc.cu) where U_1 leaves room for fewer
X tiles than two chunks of U_1 hold (rings of 6 and 7), many slices a CTA.

Small integers, so that every sum is exact: see test_gpu_residual_edges.py."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R", [((128, 512, 600), 64), ((64, 385, 450), 49), ((132, 448, 300), 64),
                                    ((36, 500, 15, 20), 60), ((128, 449, 310), 51)])
def test_residual_with_a_short_ring(cd, dims, R):
    rng = np.random.default_rng(sum(dims) + R)
    facs = [rng.integers(-2, 3, d * R).astype(np.float32) for d in dims]
    # the same slices by matrix products: integers, exact in FP32 too
    mats = [f.reshape(R, d) for f, d in zip(facs, dims)]
    kr = mats[1].T
    for m in mats[2:]:
        kr = (m.T[:, None, :] * kr[None, :, :]).reshape(-1, R)
    e = rng.integers(-1, 2, (kr.shape[0], dims[0])).astype(np.float32)
    X = kr @ mats[0] + e
    dX = torch.from_numpy(X.reshape(-1)).cuda()
    dU = [torch.from_numpy(f).cuda() for f in facs]
    for _ in range(3):
        r2, x2 = cd.cp_residual(dX, dims, dU, R)
        assert r2 == float(np.sum(e.astype(np.float64) ** 2))
        assert x2 == float(np.sum(X.astype(np.float64) ** 2))


def test_residual_ring_sizes_agree_with_the_oracle(cd):
    dims, R = (128, 400, 20), 64
    rng = np.random.default_rng(3)
    facs = [rng.integers(-2, 3, d * R).astype(np.float32) for d in dims]
    X = oracle.gencp(dims, [f.astype(np.float64) for f in facs], R)
    r2, x2 = cd.cp_residual(torch.from_numpy(X.astype(np.float32)).cuda(), dims, [torch.from_numpy(f).cuda() for f in facs], R)
    assert r2 == 0.0 and x2 == float(np.sum(X * X))

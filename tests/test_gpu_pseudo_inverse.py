"""The pseudo-inverse of a singular Gram product (solve.cu's Jacobi fallback)
at the edges of its three kernels -- one warp up to R = 16, 256 threads up to
64, 512 above -- and at odd R, whose round robin has a dummy.

Tolerance: the eigenvalues kept lie in [1, 2] and the others are rounding, so
the pseudo-inverse's condition is at most 2; Jacobi makes at most 60 sweeps of
R rounds of 2 rotations, each off by at most 2 eps of the matrix's norm:
2 x 60 x 2 x 2 R eps = 480 R eps (relative Frobenius).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [2, 3, 15, 16, 17, 63, 64, 65, 129])
def test_pseudo_inverse_of_a_singular_product(cd, R):
    rng = np.random.default_rng(R)
    k = max(1, R // 2)
    q, _ = np.linalg.qr(rng.standard_normal((R, R)))
    lam = rng.uniform(1.0, 2.0, k)
    V = (q[:, :k] * lam) @ q[:, :k].T
    want = (q[:, :k] / lam) @ q[:, :k].T
    # V = (2 V) o (1/2): the Grams of modes 0 and 2, mode 1 left out
    grams = [torch.from_numpy(np.ascontiguousarray(g)).cuda()
             for g in (2.0 * V, rng.standard_normal((R, R)), np.full((R, R), 0.5))]
    work = torch.zeros(3 * R * R + 2, dtype=torch.float64, device="cuda")
    cd.cp_normal_inverse(R, grams, 1, work)
    torch.cuda.synchronize()
    got = work[:R * R].cpu().numpy().reshape(R, R)
    assert np.linalg.norm(got - want) <= 480 * R * 2.2e-16 * np.linalg.norm(want)

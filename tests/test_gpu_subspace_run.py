"""The subspace iteration in one launch (subspace.cu k_si_run_cl) at the edges
of its layout: n below and not a multiple of the cluster's eight row blocks or
of the 8 x 8 x 4 tiles, r at each side of a multiple of 8 (and odd: a Jacobi
dummy), the largest n of each width and the next, which takes the kernels of
one launch a step; both starts.

The planted spectrum has lambda_{r+1} / lambda_r <= 0.3 and converges until
the squared sines of the subspace's angles sum to less than 1e-13 r, one more
step after that: the subspace is off by its FP32 output, 2^-24 per entry, at
most sqrt(n r) 6e-8 in the Frobenius norm twice (U U^T), and the Ritz vectors
within it by as much again over their gaps, 1 / (r - 1) here: bounds
2e-7 sqrt(n r) for U U^T and U^T U, and 2e-7 sqrt(n) for the residuals.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r", [
    (1, 1), (5, 2), (8, 8), (9, 3), (63, 7), (64, 9), (100, 16), (129, 17), (150, 24), (131, 25), (192, 31), (200, 32),
    (320, 8), (321, 8), (272, 16), (273, 16), (248, 24), (249, 24), (216, 32), (217, 32)])
@pytest.mark.parametrize("warm", [False, True])
def test_single_launch_iteration(cd, n, r, warm):
    rng = np.random.default_rng(100 * n + r)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.concatenate([np.linspace(1.0, 2.0, r), 0.3 * rng.random(n - r)])
    G = (Q * lam) @ Q.T
    G = 0.5 * (G + G.T)
    dG = torch.from_numpy(G.reshape(-1).copy()).cuda()
    U = torch.full((n * r,), 7.0, dtype=torch.float32, device="cuda")
    u0 = None
    if warm:
        u0 = torch.from_numpy((Q[:, :r] + 1e-2 * rng.standard_normal((n, r))).reshape(-1, order="F")
                              .astype(np.float32)).cuda()
    assert cd.syev_top(dG, n, r, U, u0) == cd.OK
    torch.cuda.synchronize()
    got = U.cpu().numpy().reshape(n, r, order="F").astype(np.float64)
    W = Q[:, :r]
    assert np.linalg.norm(got @ got.T - W @ W.T) <= 2e-7 * np.sqrt(n * r)
    assert np.linalg.norm(got.T @ got - np.eye(r)) <= 2e-7 * np.sqrt(n * r)
    ritz = np.einsum("ij,ik,kj->j", got, G, got)
    assert np.all(np.diff(ritz) >= -1e-6)
    assert np.linalg.norm(G @ got - got * ritz, axis=0).max() <= 2e-7 * np.sqrt(n) * 2.0

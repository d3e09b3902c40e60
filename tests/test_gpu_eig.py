"""The FP64 block Jacobi eigensolver at the edges of its 32 x 32 pair blocks
(sizes around multiples of 16 and 32), on spread, clustered and repeated
spectra, against numpy's eigh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Backward error of a Jacobi sweep: each of the O(10) sweeps of n - 1
# rotations leaves a few eps relative to ||A||; the outer stop is
# max(4 n eps, 1.3e-13).
TOL = 5e-12


def _solve(cd, torch, A):
    n = A.shape[0]
    G = torch.from_numpy(np.ascontiguousarray(A)).cuda().reshape(-1)
    W = torch.empty(n, device="cuda", dtype=torch.float64)
    V = torch.empty(n * n, device="cuda", dtype=torch.float64)
    assert cd.syev_jacobi(G, n, W, V) == cd.OK
    return W.cpu().numpy(), V.cpu().numpy().reshape(n, n).T


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 65, 97, 161])
@pytest.mark.parametrize("kind", ["spread", "clustered", "low_rank"])
def test_jacobi_eigenpairs(cd, dev, n, kind):
    import torch
    rng = np.random.default_rng(n)
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    w = {"spread": 10.0 ** rng.uniform(-6, 6, n), "clustered": 1.0 + 1e-9 * rng.standard_normal(n),
         "low_rank": np.where(np.arange(n) < max(1, n // 4), rng.uniform(1, 2, n), 0.0)}[kind]
    A = (Q * w) @ Q.T
    A = 0.5 * (A + A.T)
    W, V = _solve(cd, torch, A)
    norm = np.linalg.norm(A)
    assert np.all(np.diff(W) >= 0)
    assert np.abs(W - np.linalg.eigvalsh(A)).max() <= TOL * norm
    assert np.linalg.norm(A @ V - V * W) <= TOL * norm
    assert np.abs(V.T @ V - np.eye(n)).max() <= TOL


def test_jacobi_sort_is_stable(cd, dev):
    """A diagonal matrix needs no rotation: V is the permutation that sorts
    it, equal eigenvalues (and -0, +0) in their original order."""
    import torch
    d = np.array([2.0, 1.0, 2.0, 0.0, -0.0, 1.0, 3.0] * 30)
    n = d.size
    W, V = _solve(cd, torch, np.diag(d))
    order = np.argsort(d, kind="stable")
    assert np.array_equal(W, d[order])
    assert np.array_equal(V, np.eye(n)[:, order])

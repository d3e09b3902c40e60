"""The signs of the leading eigenvectors on the tensor-core Tucker path, where a
mode's extent is small against its rank (4 r > n: one product a step of the
subspace iteration): those of the iteration restated here in FP64 -- hashed
Gaussian start, CholeskyQR twice a step, the gap's stop and two more steps,
Rayleigh-Ritz by cyclic Jacobi."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _start(n, r):
    def mix(z):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    e = np.arange(n * r, dtype=np.uint64)
    u1 = 1.0 - (mix(2 * e + np.uint64(0x51)) >> np.uint64(11)).astype(float) / 2.0 ** 53
    u2 = (mix(2 * e + np.uint64(0x52)) >> np.uint64(11)).astype(float) / 2.0 ** 53
    return (np.sqrt(-2 * np.log(u1)) * np.cos(2 * np.pi * u2)).reshape(r, n).T


def _orth(Y):
    for _ in range(2):
        Y = np.linalg.solve(np.linalg.cholesky(Y.T @ Y), Y.T).T
    return Y


def _jacobi(H):
    r = H.shape[0]
    m = (r + 1) & ~1
    H, W = 0.5 * (H + H.T), np.eye(r)
    for _ in range(40):
        if (H ** 2).sum() - (np.diag(H) ** 2).sum() <= 1e-26 * (H ** 2).sum():
            break
        for rd in range(m - 1):
            J = np.eye(r)
            for k in range(m // 2):
                a, b = (m - 1, rd % (m - 1)) if k == 0 else ((rd + k) % (m - 1), (rd + m - 1 - k) % (m - 1))
                p, q = min(a, b), max(a, b)
                if q < r and abs(H[p, q]) > 1e-100:
                    th = (H[q, q] - H[p, p]) / (2 * H[p, q])
                    t = (1.0 if th >= 0 else -1.0) / (abs(th) + np.sqrt(th * th + 1))
                    c = 1 / np.sqrt(t * t + 1)
                    J[p, p], J[q, q], J[p, q], J[q, p] = c, c, t * c, -t * c
            H, W = J.T @ H @ J, W @ J
    return W[:, np.argsort(np.diag(H), kind="stable")]


def _top(G, r):
    V, extra = _orth(_start(len(G), r)), -1
    for _ in range(300):
        Y = _orth(G @ V)
        gap, V = r - np.sum((V.T @ Y) ** 2), Y
        if extra < 0 and gap < 1e-13 * r:
            extra = 2
        if extra == 0:
            return V @ _jacobi(V.T @ (G @ V))
        extra -= extra > 0
    raise AssertionError("not converged")


@pytest.mark.parametrize("seed", range(8))
def test_signs_where_the_rank_is_over_a_quarter(cd, dev, seed):
    import torch
    dims, ranks = (32, 40, 48), (10, 12, 14)
    rng = np.random.default_rng(seed)
    X = rng.standard_normal(ranks)
    for m, (d, r) in enumerate(zip(dims, ranks)):
        Q = np.linalg.qr(rng.standard_normal((d, r)))[0] * np.linspace(1.0, 0.4, r)
        X = np.moveaxis(np.tensordot(Q, X, axes=(1, m)), 0, m)
    X += 1e-2 * np.linalg.norm(X) / np.sqrt(X.size) * rng.standard_normal(dims)
    core = torch.empty(int(np.prod(ranks)), device="cuda")
    U = [torch.empty(d * r, device="cuda") for d, r in zip(dims, ranks)]
    cd.tucker_hosvd(torch.from_numpy(X.astype(np.float32).reshape(-1, order="F")).cuda(), dims, ranks, core, U,
                    cd.PREC_BF16X3)
    for m, (d, r) in enumerate(zip(dims, ranks)):
        assert 3 * d * r + 8 <= d * d < 4 * d * r + 8
        T = np.moveaxis(X.astype(np.float32).astype(float), m, 0).reshape(d, -1)
        want, got = _top(T @ T.T, r), U[m].cpu().numpy().reshape(r, d).T
        # (noise of 1e-2 keeps the trailing eigenvalues, and with them the number
        # of steps, clear of the Gram's BF16x3 rounding)
        assert np.all(np.sum(want * got, axis=0) > 0.9), m

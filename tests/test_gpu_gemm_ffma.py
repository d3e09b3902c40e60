"""Mode products and unfolding Grams in FP32 at the edges of the FFMA GEMM's
tiles and of the rule that chooses it (128-row tiles, column tiles of 8 to 64,
32-deep stages, two-level rows, 16- and 4-byte copies, contractions around 64,
96 and 512) -- against FP64 on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((1, 1), 1), ((64, 300), 5), ((300, 64), 8), ((33, 96, 29), 9), ((128, 64, 32), 16), ((130, 65, 31), 17),
          ((5, 300, 70), 32), ((4, 97, 50), 33), ((127, 95, 40), 64), ((96, 40, 90), 65), ((2, 3, 600), 40),
          ((9, 8, 70, 66), 20), ((63, 64, 64), 130)]


def _upload(torch, x, offset):
    buf = torch.empty(x.size + 4, device="cuda")
    d = buf[offset: offset + x.size]
    d.copy_(torch.from_numpy(x))
    return d


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dims,J", SHAPES)
def test_mode_product_edges(cd, dev, dims, J, offset):
    import torch
    rng = np.random.default_rng(sum(dims) + J)
    X = rng.standard_normal(int(np.prod(dims))).astype(np.float32)
    dX = _upload(torch, X, offset)
    for mode, d in enumerate(dims):
        W = rng.standard_normal((d, J)).astype(np.float32)  # column-major J x d
        T = np.moveaxis(X.astype(np.float64).reshape(dims, order="F"), mode, 0)

        def fold(A):
            Y = np.tensordot(A, np.abs(T) if A is aW else T, axes=(0, 0))
            return np.moveaxis(Y, 0, mode).reshape(-1, order="F")

        aW = np.abs(W.astype(np.float64))
        want, scale = fold(W.astype(np.float64)), fold(aW)
        out = torch.full((want.size,), 7.0, device="cuda")
        cd.mode_product(dX, dims, mode, torch.from_numpy(W.reshape(-1)).cuda(), J, out)
        # componentwise n eps |W||X| at 64 steps of a chain in effect
        assert np.all(np.abs(out.cpu().numpy() - want) <= 64 * 2.0 ** -24 * scale)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1), (64, 511), (33, 31, 29), (128, 8, 64), (130, 66, 9), (40, 50, 60), (5, 6, 7, 80)])
def test_unfold_gram_edges(cd, dev, dims, offset):
    import torch
    rng = np.random.default_rng(sum(dims))
    X = rng.standard_normal(int(np.prod(dims))).astype(np.float32)
    dX = _upload(torch, X, offset)
    for mode, d in enumerate(dims):
        T = np.moveaxis(X.astype(np.float64).reshape(dims, order="F"), mode, 0).reshape(d, -1)
        G = torch.empty(d * d, device="cuda", dtype=torch.float64)
        cd.unfold_gram(dX, dims, mode, G)
        err = np.abs(G.cpu().numpy().reshape(d, d) - T @ T.T)
        assert np.all(err <= 64 * 2.0 ** -24 * (np.abs(T) @ np.abs(T).T))

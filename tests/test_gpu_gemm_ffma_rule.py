"""FP32 mode products and unfolding Grams at each side of the rules between the
FFMA tile and the 64 x 64 tile: more than 32 columns over enough tiles for the
GPU, few tiles, short inner contractions, and split ranges fitted to the SMs.
Small integers, whose sums are exact in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,J", [((31, 77, 500), 128), ((150, 150, 150), 64), ((151, 149, 131), 47), ((70, 70, 70), 24),
                                    ((200, 100, 101), 200), ((65, 97, 33, 9), 72), ((500, 64, 80), 64)])
def test_mode_products(cd, dev, dims, J):
    import torch
    rng = np.random.default_rng(sum(dims) + J)
    X = torch.from_numpy(rng.integers(-2, 3, int(np.prod(dims))).astype(np.float32)).cuda()
    T = X.double().reshape(tuple(reversed(dims)))  # axes run slowest mode first
    for mode, d in enumerate(dims):
        W = torch.from_numpy(rng.integers(-2, 3, (d, J)).astype(np.float32)).cuda()  # column-major J x d
        axis = len(dims) - 1 - mode
        want = torch.movedim(torch.tensordot(T, W.double(), dims=([axis], [0])), -1, axis)
        out = torch.full((want.numel(),), 7.0, device="cuda")
        cd.mode_product(X, dims, mode, W.reshape(-1), J, out)
        assert torch.equal(out.double(), want.reshape(-1)), mode


@pytest.mark.parametrize("dims", [(2, 300, 100), (5, 130, 300), (6, 130, 300), (7, 130, 300), (100, 100, 100),
                                  (787, 60, 9), (130, 999, 6)])
def test_unfolding_grams(cd, dev, dims):
    import torch
    rng = np.random.default_rng(sum(dims))
    X = torch.from_numpy(rng.integers(-2, 3, int(np.prod(dims))).astype(np.float32)).cuda()
    T = X.double().reshape(tuple(reversed(dims)))
    for mode, d in enumerate(dims):
        M = torch.movedim(T, len(dims) - 1 - mode, 0).reshape(d, -1)
        G = torch.empty(d * d, device="cuda", dtype=torch.float64)
        cd.unfold_gram(X, dims, mode, G)
        assert torch.equal(G.reshape(d, d), M @ M.T), mode

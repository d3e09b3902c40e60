"""The FP64 MTTKRP at the edges of its tiles: 128-row tiles, 16-deep stages
that end with a row block of the fastest factor, the rank groups of 8 (up to
64 a CTA, and above), 16- and 8-byte copies, 2nd- to 6th-order tensors, and an
infinity beside a ragged block -- against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((1, 1), 1), ((129, 33), 9), ((1, 5, 1), 3), ((3, 2, 2), 4), ((33, 31, 29), 5), ((128, 16, 32), 8),
          ((5, 300, 7), 16), ((260, 3, 50), 17), ((127, 129, 4), 33), ((64, 64, 34), 48), ((36, 20, 40), 65),
          ((9, 8, 7, 6), 20), ((12, 5, 3, 4, 7), 11), ((2, 3, 2, 3, 2, 3), 6), ((31, 1, 77), 28)]


def _want(X, dims, U, mode):
    T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
    kr = None
    for m, u in enumerate(U):
        if m != mode:
            kr = u.T if kr is None else (u.T[:, None, :] * kr[None, :, :]).reshape(-1, u.shape[0])
    return T @ kr, np.abs(T) @ np.abs(kr)


def _run(cd, torch, X, dims, U, R, mode, offset):
    buf = torch.empty(X.size + 2, device="cuda", dtype=torch.float64)
    dX = buf[offset: offset + X.size]
    dX.copy_(torch.from_numpy(X))
    out = torch.full((dims[mode] * R,), 7.0, device="cuda", dtype=torch.float64)
    cd.mttkrp_f64(dX, dims, [torch.from_numpy(np.ascontiguousarray(u).reshape(-1)).cuda() for u in U], mode, R, out)
    return out.cpu().numpy().reshape(dims[mode], R, order="F")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dims,R", SHAPES)
def test_f64_edges(cd, dev, dims, R, offset):
    import torch
    rng = np.random.default_rng(sum(dims) + R)
    X = rng.standard_normal(int(np.prod(dims)))
    U = [rng.standard_normal((R, d)) for d in dims]
    for mode in range(len(dims)):
        want, scale = _want(X, dims, U, mode)
        got = _run(cd, torch, X, dims, U, R, mode, offset)
        # componentwise n eps |X||KR| at 64 steps (both sides round)
        assert np.all(np.abs(got - want) <= 64 * 2.0 ** -53 * scale)


def test_f64_infinities_stay_in_their_rows(cd, dev):
    import torch
    dims, R = (38, 37, 5), 6
    rng = np.random.default_rng(3)
    X = rng.standard_normal(int(np.prod(dims)))
    X[3 + 38 * (36 + 37 * 2)] = np.inf
    U = [rng.random((R, d)) + 0.5 for d in dims]
    for mode, row in enumerate((3, 36, 2)):
        got = _run(cd, torch, X, dims, U, R, mode, 0)
        assert np.all(np.isposinf(got[row]))
        assert np.all(np.isfinite(np.delete(got, row, axis=0)))

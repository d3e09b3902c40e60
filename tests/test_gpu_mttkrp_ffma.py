"""The FP32 FFMA MTTKRP at the edges of its tiles: 128-row tiles, 32-deep
stages that end with a row block of the fastest factor, the rank tiles
(1-4, 5-8, 9-16, 17-32, 33-64, above), 16- and 4-byte copies (extents,
alignment), 2nd- to 6th-order tensors, operand rounding, and infinities
beside a ragged block -- against FP64 on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((1, 1), 1), ((129, 33), 9), ((1, 5, 1), 3), ((3, 2, 2), 4), ((33, 31, 29), 5), ((128, 32, 32), 8),
          ((5, 300, 7), 16), ((260, 3, 50), 17), ((127, 129, 4), 33), ((64, 64, 64), 64), ((36, 20, 40), 65),
          ((30, 22, 20), 130), ((9, 8, 7, 6), 20), ((12, 5, 3, 4, 7), 11), ((2, 3, 2, 3, 2, 3), 6), ((31, 1, 77), 28)]


def _case(dims, R, seed, offset):
    """Data whose X sits `offset` floats past a 16-byte boundary."""
    import torch
    rng = np.random.default_rng(seed)
    X = rng.standard_normal(int(np.prod(dims))).astype(np.float32)
    U = [rng.standard_normal((R, d)).astype(np.float32) for d in dims]
    buf = torch.empty(X.size + 4, device="cuda")
    dX = buf[offset: offset + X.size]
    dX.copy_(torch.from_numpy(X))
    return X, U, dX, [torch.from_numpy(u.reshape(-1)).cuda() for u in U]


def _kr(U):
    kr = U[0].T
    for u in U[1:]:
        kr = (u.T[:, None, :] * kr[None, :, :]).reshape(-1, kr.shape[1])
    return kr


def _want(X, dims, U, mode):
    """(M, |X| |KR|): the product in FP64, and the same of absolute values."""
    T = np.moveaxis(X.astype(np.float64).reshape(dims, order="F"), mode, 0)
    T = T.reshape(dims[mode], -1, order="F")
    kr = _kr([u.astype(np.float64) for m, u in enumerate(U) if m != mode])
    return T @ kr, np.abs(T) @ np.abs(kr)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dims,R", SHAPES)
def test_ffma_edges(cd, dev, dims, R, offset):
    import torch
    X, U, dX, dU = _case(dims, R, sum(dims) + R, offset)
    for mode in range(len(dims)):
        want, scale = _want(X, dims, U, mode)
        out = torch.full((dims[mode] * R,), 7.0, device="cuda")
        cd.mttkrp(dX, dims, dU, mode, R, out, cd.PREC_FP32)
        got = out.cpu().numpy().reshape(dims[mode], R, order="F")
        # N roundings of the product entries and the FP32 chains of a split:
        # componentwise n eps |X||KR|, far fewer than 64 steps deep in effect
        assert np.all(np.abs(got - want) <= 64 * 2.0 ** -24 * scale)


@pytest.mark.parametrize("dims,R", [((33, 31, 29), 5), ((50, 60, 70), 130), ((7, 9, 11, 13), 20)])
@pytest.mark.parametrize("prec", ["fp16", "bf16"])
def test_ffma_rounds_operands(cd, dev, dims, R, prec):
    """X and each Khatri-Rao entry (one FP32 product) rounded first."""
    import torch
    X, U, dX, dU = _case(dims, R, 5, 1)

    def rnd(a):
        t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32))
        return t.to(torch.float16 if prec == "fp16" else torch.bfloat16).float().numpy().astype(np.float64)

    for mode in range(len(dims)):
        T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
        kr = _kr([u for m, u in enumerate(U) if m != mode])
        want = rnd(T) @ rnd(kr)
        scale = np.abs(rnd(T)) @ np.abs(rnd(kr))
        out = torch.empty(dims[mode] * R, device="cuda")
        cd.mttkrp(dX, dims, dU, mode, R, out, cd.PRECISIONS[prec])
        got = out.cpu().numpy().reshape(dims[mode], R, order="F")
        # three or more factors may be multiplied in another order than here:
        # a product one FP32 ulp apart can round to the neighbouring 16-bit
        # value, for few entries
        assert np.linalg.norm(got - want) <= 1e-4 * np.linalg.norm(scale)


def test_ffma_infinities_stay_in_their_rows(cd, dev):
    """An infinite entry of X makes its own row of M infinite or NaN, no other
    row, and stays infinite where the Khatri-Rao value is finite: nothing past
    a row block's end is multiplied by it."""
    import torch
    dims, R = (38, 37, 5), 6
    X, U, dX, dU = _case(dims, R, 11, 0)
    U = [np.abs(u) + 0.5 for u in U]
    dU = [torch.from_numpy(u.reshape(-1)).cuda() for u in U]
    X[3 + 38 * (36 + 37 * 2)] = np.inf
    dX.copy_(torch.from_numpy(X))
    for mode, row in enumerate((3, 36, 2)):
        out = torch.empty(dims[mode] * R, device="cuda")
        cd.mttkrp(dX, dims, dU, mode, R, out, cd.PREC_FP32)
        got = out.cpu().numpy().reshape(dims[mode], R, order="F")
        assert np.all(np.isposinf(got[row]))
        assert np.all(np.isfinite(np.delete(got, row, axis=0)))

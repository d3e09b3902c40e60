"""The one-launch MTTKRP of small tensors (plain FP32, CUD_PREC_FP32 and
CUD_PREC_DEFAULT) at the edges of its tiles: 4 rows x 8 ranks a cluster,
clusters of 1 to 8 CTAs, contractions below and above a thread each, 16-byte
and scalar reads; and the rule that hands DEFAULT to FP32 or to the tensor
cores -- against FP64 on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((1, 1), 1), ((5, 3), 2), ((3, 255), 7), ((4, 513), 9), ((7, 40, 50), 8), ((48, 40, 36), 8), ((6, 5, 4, 3), 17),
          ((2, 3, 2, 3, 2), 5), ((30, 64, 70), 33), ((1, 128, 127), 64), ((600, 9, 11), 3), ((64, 64, 64), 32)]


@pytest.mark.parametrize("prec", ["fp32", "default"])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("dims,R", SHAPES)
def test_small_edges(cd, dev, dims, R, offset, prec):
    import torch
    rng = np.random.default_rng(sum(dims) + R)
    X = rng.standard_normal(int(np.prod(dims))).astype(np.float32)
    U = [rng.standard_normal((R, d)).astype(np.float32) for d in dims]
    buf = torch.empty(X.size + 4, device="cuda")
    dX = buf[offset: offset + X.size]
    dX.copy_(torch.from_numpy(X))
    dU = [torch.from_numpy(u.reshape(-1)).cuda() for u in U]
    for mode in range(len(dims)):
        assert cd.mttkrp_path(dims, mode, R, cd.PRECISIONS[prec]) == "cuda-core"
        T = np.moveaxis(X.astype(np.float64).reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
        kr = None
        for m, u in enumerate(U):
            if m != mode:
                u = u.astype(np.float64)
                kr = u.T if kr is None else (u.T[:, None, :] * kr[None, :, :]).reshape(-1, R)
        out = torch.full((dims[mode] * R,), 7.0, device="cuda")
        cd.mttkrp(dX, dims, dU, mode, R, out, cd.PRECISIONS[prec])
        got = out.cpu().numpy().reshape(dims[mode], R, order="F")
        # n eps |X||KR| for the few roundings of a thread's chain and the tree
        assert np.all(np.abs(got - T @ kr) <= 32 * 2.0 ** -24 * (np.abs(T) @ np.abs(kr)))


def test_default_takes_the_faster_path(cd, dev):
    assert cd.mttkrp_path((512, 512, 512), 0, 64) == "tensor-core"
    assert cd.mttkrp_path((96, 96, 96, 96), 2, 32) == "tensor-core"
    assert cd.mttkrp_path((200, 200, 200), 1, 16) == "cuda-core"       # Khatri-Rao rows would be built per stage
    assert cd.mttkrp_path((200, 200, 200), 1, 16, cd.PREC_BF16X3) == "tensor-core"
    assert cd.mttkrp_path((128, 128, 128), 0, 16) == "cuda-core"       # too little work

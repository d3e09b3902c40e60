"""The split reduce behind the MTTKRP kernels at each side of its rule: many
splits of few outputs, outputs around the limit of a wave, and fewer splits
than lanes -- small integers, whose sums are exact in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R", [((160, 160, 40), 59), ((160, 160, 40), 60), ((20, 300, 90), 9), ((5000, 30, 20), 20),
                                    ((40000, 12, 12), 5)])
@pytest.mark.parametrize("prec", ["fp32", "bf16x3", "f64"])
def test_exact_sums(cd, dev, dims, R, prec):
    import torch
    rng = np.random.default_rng(R + dims[0])
    X = rng.integers(-2, 3, int(np.prod(dims))).astype(np.float64)
    U = [rng.integers(-1, 2, (R, d)).astype(np.float64) for d in dims]
    dtype = torch.float64 if prec == "f64" else torch.float32
    dX = torch.from_numpy(X).to(dtype).cuda()
    dU = [torch.from_numpy(u.reshape(-1)).to(dtype).cuda() for u in U]
    T = torch.from_numpy(X.reshape(dims, order="F"))
    for mode in range(3):
        a, b = [m for m in range(3) if m != mode]
        want = torch.einsum("qab,ra,rb->qr", T.permute(mode, a, b), torch.from_numpy(U[a]), torch.from_numpy(U[b]))
        out = torch.empty(dims[mode] * R, device="cuda", dtype=dtype)
        if prec == "f64":
            cd.mttkrp_f64(dX, dims, dU, mode, R, out)
        else:
            cd.mttkrp(dX, dims, dU, mode, R, out, cd.PRECISIONS[prec])
        assert torch.equal(out.cpu().double().reshape(R, dims[mode]).T, want)

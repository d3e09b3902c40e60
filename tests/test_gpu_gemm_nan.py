"""A NaN accumulator -- a NaN operand, or a CTA whose bounded wait ran out --
must reach the outputs of a BF16 GEMM through the ReLU, in every epilogue: the
tiles of 128 and 256 columns, a split contraction, and the skinny kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(200, 100, 128), (300, 520, 256), (256, 256, 65536), (40000, 16, 128)])
def test_nan_passes_the_relu(cd, M, N, K):
    g = torch.Generator().manual_seed(M + N)
    A = torch.randint(-2, 3, (M, K), generator=g).to(torch.bfloat16)
    B = torch.randint(-2, 3, (N, K), generator=g).to(torch.bfloat16)
    A[M // 2, K - 1] = float("nan")
    C = torch.zeros((M, N), device="cuda")
    H = torch.zeros((M, N), device="cuda", dtype=torch.bfloat16)
    cd.gemm_bf16(A.cuda(), B.cuda(), relu=True, out_f32=C, out_bf16=H)
    want = torch.relu(A.float() @ B.float().T)  # integers: exact in FP32
    rest = [m for m in range(M) if m != M // 2]
    for got, ref in ((C.cpu(), want), (H.cpu(), want.to(torch.bfloat16))):
        assert torch.all(torch.isnan(got[M // 2]))
        assert torch.equal(got[rest], ref[rest])

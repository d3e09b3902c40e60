"""Products queued one behind the other (gemm_tc.cu launches each kernel
programmatically): every product adds to the same output, through one
workspace, so each depends on the one before it -- with contraction splits at
each side of the 16 partials that the split sum reads at a time, and the
skinny kernel.  Integers: exact.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,Ks", [
    (64, 64, [256 * s for s in (1, 2, 15, 16, 17, 33, 74)]),   # one tile: K / 256 splits
    (200, 300, [64, 8192, 256, 5000, 72]),
    (40000, 16, [128, 512, 64])])                              # skinny
def test_chained_products(cd, M, N, Ks):
    g = torch.Generator().manual_seed(M + N)
    ops = [(torch.randint(-2, 3, (M, K), generator=g), torch.randint(-2, 3, (N, K), generator=g)) for K in Ks]
    want = sum((a.float() @ b.float().T for a, b in ops), torch.zeros(M, N))  # exact: |sums| < 2^24
    dev = [(a.to(torch.bfloat16).cuda(), b.to(torch.bfloat16).cuda()) for a, b in ops]
    for rep in range(5):
        C = torch.zeros((M, N), device="cuda")
        for a, b in dev:
            cd.gemm_bf16(a, b, out_f32=C, accumulate=True)
        torch.cuda.synchronize()
        assert torch.equal(C.cpu(), want)

"""The tensor-core CP residual (residual_tc.cu) at the edges of its tiles: rows
that end in each quarter of a 128-row tile, U_1 at each side of a 32-column X
tile and of a 128-column chunk, ranks at each side of 16, 32 and 48, fewer and
more slices than CTAs, orders 3 to 5, and an X that TMA cannot read (another
kernel).

Small integers: every factor product, reconstructed entry, square and sum is
an integer that BF16, FP32 and FP64 hold exactly (|U| <= 2, so |c_k| <= 8 and
|A'| <= 16; |X - Xh| <= 1; |Xh| <= 64 * 32 < 2^24), so the sums are exact.
"""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R", [
    ((4, 1, 1), 1), ((32, 31, 3), 16), ((36, 32, 5), 17), ((64, 33, 200), 32), ((68, 96, 7), 33), ((100, 97, 3), 48),
    ((128, 127, 149), 64), ((132, 128, 9), 49), ((256, 129, 4), 16), ((260, 300, 3), 20), ((40, 20, 6, 5), 12),
    ((12, 160, 2, 3, 4), 31)])
@pytest.mark.parametrize("shift", [0, 1])
def test_residual_at_tile_edges(cd, dims, R, shift):
    rng = np.random.default_rng(sum(dims) + R)
    facs = [rng.integers(-2, 3, d * R).astype(np.float32) for d in dims]
    rec = oracle.gencp(dims, [f.astype(np.float64) for f in facs], R)
    e = rng.integers(-1, 2, rec.size).astype(np.float64)
    X = rec + e
    dX = torch.from_numpy(np.concatenate([np.zeros(shift), X]).astype(np.float32)).cuda()[shift:]
    dU = [torch.from_numpy(f).cuda() for f in facs]
    r2, x2 = cd.cp_residual(dX, dims, dU, R)
    assert r2 == float(np.sum(e * e))
    assert x2 == float(np.sum(X * X))
